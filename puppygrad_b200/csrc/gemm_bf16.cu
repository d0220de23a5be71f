// BF16 tensor-core products of the layered models (sm_100a): tcgen05.mma kind::f16, operands staged by TMA with
// 128-byte swizzle, FP32 accumulators in tensor memory, warp-specialised roles, bounded waits.
//
//   tc_gemm_bf16_kernel       out[m, n] = x[m, k] . w[n, k]^T for whole portions of prompts: 128 x BN tiles of the
//                             output, persistent, results leave through shared memory by TMA stores
//   tc_gemm_bf16_rows_kernel  the same product for at most 64 rows (a decode step): 128 weight rows are the wide operand,
//                             read in 16 KB tiles, k is cut over a thread-block cluster whose blocks exchange partial sums through
//                             distributed shared memory, and the weight stream starts before the dependency wait
//
// On an expired wait a kernel raises the error flag, stops issuing work, still frees its tensor memory and returns.
#include <algorithm>

#include "device_util.cuh"
#include "layered_kernels.cuh"
#include "tc_common.cuh"

namespace pg {
namespace {

constexpr int KB = 64;  // BF16 elements per k block: one 128-byte swizzle row

// z * Phi(z) of two values for results that are rounded to BF16 next. Phi(z) - 1/2 = z P(2 z^2 / 4.5^2 - 1) on
// [-4.5, 4.5] with a degree-9 weighted least-squares fit of (Phi(z) - 1/2) / z on Chebyshev nodes; beyond that range Phi
// is taken at its end. Absolute error below 1e-5 inside and 5e-5 outside.
__device__ __forceinline__ void gelu_erf_pair(float& x, float& y) {
  constexpr float C[10] = {1.569053008e-01f, -7.718336822e-02f, 5.467184018e-02f, -4.029580498e-02f, 2.862407447e-02f,
                           -1.815922087e-02f, 1.014016557e-02f, -6.682699045e-03f, 4.655552699e-03f, -1.565833704e-03f};
  const float cx = fminf(fmaxf(x, -4.5f), 4.5f), cy = fminf(fmaxf(y, -4.5f), 4.5f);
  const unsigned long long c2 = pack2(cx, cy), zero = pack2(0.f, 0.f);
  const unsigned long long t = fma2(fma2(c2, c2, zero), pack2(2.f / 20.25f, 2.f / 20.25f), pack2(-1.f, -1.f));
  unsigned long long p = pack2(C[9], C[9]);
#pragma unroll
  for (int i = 8; i >= 0; --i) p = fma2(p, t, pack2(C[i], C[i]));
  p = fma2(p, c2, pack2(0.5f, 0.5f));
  float px, py;
  unpack2(p, px, py);
  x *= px;
  y *= py;
}

__device__ __forceinline__ float exp2_fast(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// xIELU for results that are rounded to BF16 next: e^z - 1 - z is off by less than 1e-6 here, far below z / 2 wherever that
// rounds to a BF16 of its own.
__device__ __forceinline__ float xielu_fast(float z, float a, float b) {
  const float e = exp2_fast(fminf(z, 0.f) * 1.4426950408889634f) - 1.f - z;
  return fmaf(0.5f, z, z > 0.f ? a * z * z : b * e);
}
__device__ __forceinline__ void activate_pair(const ActArgs& act, float& x, float& y) {
  if (act.kind == ACT_GELU_ERF) {
    gelu_erf_pair(x, y);
  } else if (act.kind == ACT_XIELU) {
    x = xielu_fast(x, act.a, act.b);
    y = xielu_fast(y, act.a, act.b);
  }
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y, const void* smem_src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x), "r"(y),
               "r"(smem_u32(smem_src))
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

template <int BN>
struct BfSmem {
  static constexpr int STAGES = (BN == 256) ? 4 : 6;
  static constexpr int A_BYTES = TILE_M * KB * 2, B_BYTES = BN * KB * 2;
  static constexpr int BOX_BYTES = 32 * 128;            // 32 rows of 128 bytes: one store box
  static constexpr int EPI_BYTES = 4 * 2 * BOX_BYTES;   // two boxes per epilogue warp
  static constexpr size_t BYTES = (size_t)STAGES * (A_BYTES + B_BYTES) + EPI_BYTES + 1024 /*align*/ + 256 /*barriers*/;
};

enum { OUT_F32 = 0, OUT_BF16 = 1, OUT_BF16_ACT = 2 };

// Persistent over 128 x BN output tiles; two accumulators in tensor memory, so that the epilogue of a tile overlaps the
// products of the next. Warp 0 loads, warp 1 issues the MMAs and owns the tensor memory, warps 2..5 store. `tma_out`:
// map_o can be used (16-byte aligned rows); else rows are stored element by element.
template <int BN>
__global__ void __launch_bounds__(192, 1)
    tc_gemm_bf16_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                        const __grid_constant__ CUtensorMap map_o, Bf16GemmArgs a, int out_kind, int tma_out) {
  using S = BfSmem<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* smem_a = base;
  uint8_t* smem_b = base + (size_t)S::STAGES * S::A_BYTES;
  uint8_t* epi = smem_b + (size_t)S::STAGES * S::B_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(epi + S::EPI_BYTES);
  uint64_t* empty = full + S::STAGES;
  uint64_t* d_full = empty + S::STAGES;  // [2]: accumulator holds a finished tile
  uint64_t* d_empty = d_full + 2;        // [2]: the epilogue warps have read it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(d_empty + 2);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = (a.m + TILE_M - 1) / TILE_M, tiles_n = (a.n + BN - 1) / BN, tiles = tiles_n * tiles_m;
  const int nkb = (a.k + KB - 1) / KB;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&d_full[i], 1);
      mbar_init(&d_empty[i], 4);
    }
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, 2 * BN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch();
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0;  // stage counter over all tiles of this block
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int n0 = (tile % tiles_n) * BN, m0 = (tile / tiles_n) * TILE_M;
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          const uint32_t s = it % S::STAGES;
          if (it >= S::STAGES) ok = mbar_wait(&empty[s], ((it / S::STAGES) - 1) & 1, failed, a.error_flag, 1);
          if (!ok) break;
          mbar_expect_tx(&full[s], S::A_BYTES + S::B_BYTES);
          tma_load_2d(smem_a + (size_t)s * S::A_BYTES, &map_x, kb * KB, m0, &full[s]);
          tma_load_2d(smem_b + (size_t)s * S::B_BYTES, &map_w, kb * KB, n0, &full[s]);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = umma_idesc_bf16(TILE_M, BN);
      uint32_t it = 0, ti = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++ti) {
        const uint32_t buf = ti & 1;
        if (ti >= 2) ok = mbar_wait(&d_empty[buf], ((ti >> 1) - 1) & 1, failed, a.error_flag, 4);
        if (!ok) break;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + buf * BN;
        for (int kb = 0; kb < nkb && ok; ++kb, ++it) {
          const uint32_t s = it % S::STAGES;
          ok = mbar_wait(&full[s], (it / S::STAGES) & 1, failed, a.error_flag, 2);
          if (!ok) break;
          tc_fence_after();
          const uint64_t da = umma_desc_sw128(smem_a + (size_t)s * S::A_BYTES);
          const uint64_t db = umma_desc_sw128(smem_b + (size_t)s * S::B_BYTES);
#pragma unroll
          for (int k = 0; k < KB / 16; ++k)
            umma_bf16_ss(tmem_d, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb | k) != 0);
          umma_commit(&empty[s]);
        }
        if (ok) umma_commit(&d_full[buf]);
      }
    }
  } else {
    const int q = warp & 3;  // tensor-memory lane quarter of this warp
    uint8_t* boxes = epi + (size_t)(warp - 2) * 2 * S::BOX_BYTES;
    const int cols = out_kind == OUT_F32 ? 32 : 64;  // columns of one 128-byte box row
    uint32_t ti = 0, nbox = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++ti) {
      const int n0 = (tile % tiles_n) * BN, m0 = (tile / tiles_n) * TILE_M + q * 32;
      const uint32_t buf = ti & 1, tmem_d = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16);
      ok = mbar_wait(&d_full[buf], (ti >> 1) & 1, failed, a.error_flag, 3);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
#pragma unroll 1
      for (int c0 = 0; c0 < BN && n0 + c0 < a.n; c0 += cols) {
        float v[32];
        tmem_ld32(tmem_d + (uint32_t)c0, v);
        uint8_t* box = boxes + (nbox & 1) * S::BOX_BYTES;
        uint4* row = reinterpret_cast<uint4*>(box + lane * 128);
        if (tma_out) {
          if (lane == 0) bulk_wait_read<1>();  // the box's previous store has read it
          __syncwarp();
        }
        if (out_kind == OUT_F32) {
          if (tma_out) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              row[j ^ (lane & 7)] = make_uint4(__float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]), __float_as_uint(v[4 * j + 2]),
                                               __float_as_uint(v[4 * j + 3]));
          } else if (m0 + lane < a.m) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (n0 + c0 + j < a.n) a.out[(size_t)(m0 + lane) * a.ldo + n0 + c0 + j] = v[j];
          }
        } else {
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            if (half) tmem_ld32(tmem_d + (uint32_t)(c0 + 32), v);
            if (out_kind == OUT_BF16_ACT) {
#pragma unroll
              for (int j = 0; j < 32; j += 2) activate_pair(a.act, v[j], v[j + 1]);
            }
            uint32_t p[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
              p[j] = *reinterpret_cast<const uint32_t*>(&b);
            }
            if (tma_out) {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                row[(half * 4 + j) ^ (lane & 7)] = make_uint4(p[4 * j], p[4 * j + 1], p[4 * j + 2], p[4 * j + 3]);
            } else if (m0 + lane < a.m) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (n0 + c0 + half * 32 + j < a.n)
                  static_cast<__nv_bfloat16*>(a.out_h)[(size_t)(m0 + lane) * a.ldo + n0 + c0 + half * 32 + j] = __float2bfloat16_rn(v[j]);
            }
          }
        }
        if (tma_out) {
          fence_async_shared();
          __syncwarp();
          if (lane == 0) {
            if (m0 < a.m) tma_store_2d(&map_o, n0 + c0, m0, box);
            bulk_commit();
          }
          ++nbox;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&d_empty[buf]);
    }
    if (lane == 0) bulk_wait_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 2 * BN);
}

// ------------------------------------------------------------------ decode rows
// A ring of stages of ROWS weight rows and BN input rows. The ring is smaller than half an SM's shared memory: the next kernel's blocks
// find room beside the running ones and have their first weights loaded when the dependency is released.
template <int BN, int ROWS>
struct RowsSmem {
  static constexpr int A_BYTES = ROWS * KB * 2, B_BYTES = BN * KB * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;  // both multiples of 1024
  static constexpr int STAGES = ROWS == 64 ? (BN == 64 ? 6 : BN == 32 ? 8 : 9) : BN == 64 ? 4 : 5;
  static constexpr size_t BYTES = (size_t)STAGES * STAGE_BYTES + 1024 + 256;
  static_assert(ROWS * BN * 4 <= STAGES * STAGE_BYTES, "the partial sums reuse the ring");
  static_assert(2 * (BYTES + 1024) <= 228 * 1024, "two blocks on an SM");
};

__device__ __forceinline__ float4 cluster_load4(uint32_t addr, uint32_t rank) {
  uint32_t r;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(r) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// A block multiplies ROWS weight rows with the m <= BN input rows over its share of k, leaves the partial sums in its shared
// memory (where the operands were), and the blocks of the cluster each add and store an equal part of the tile, in split order.
//
// Bound by the weight stream: 64 rows, inside a step, us (and TB/s) with ROWS 128 and with 64: 2048 x 8192 in four parts 16.5 -> 14.3 (2.3),
// 14656 x 2048 in one 20.4 -> 16.3 (3.7), 9536 x 2048 21.6 -> 16.2 (2.4); 32000 x 2048, which has 250 blocks of 128, 25.6 (5.1).
template <int BN, int ROWS>
__global__ void __launch_bounds__(192, 2)
    tc_gemm_bf16_rows_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, Bf16GemmArgs a,
                             int out_kind) {
  using S = RowsSmem<BN, ROWS>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* part = reinterpret_cast<float*>(base);  // [BN][ROWS], once the products are done
  uint64_t* full = reinterpret_cast<uint64_t*>(base + (size_t)S::STAGES * S::STAGE_BYTES);
  uint64_t* empty = full + S::STAGES;
  uint64_t* d_full = empty + S::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(d_full + 1);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
  constexpr uint32_t COLS = BN < 32 ? 32 : BN;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * ROWS, split = blockIdx.y, splits = gridDim.y;
  const int nkb_all = (a.k + KB - 1) / KB, kb0 = nkb_all * split / splits, nkb = nkb_all * (split + 1) / splits - kb0;
  const int head = blockIdx.z, x0 = head * a.x_head;
  // first row of this block's part of the weight tiles, which have TILE_M rows
  const int row_tiles = ((int)gridDim.x * ROWS + TILE_M - 1) / TILE_M;
  const int wrow = ((head * row_tiles + n0 / TILE_M) * nkb_all + kb0) * TILE_M + n0 % TILE_M;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(d_full, 1);
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_d = *tmem_slot;
  pdl_launch();

  if (warp == 0) {
    if (lane == 0) {
      const int ahead = min(nkb, S::STAGES);
      for (int i = 0; i < ahead; ++i) {  // weights do not depend on the previous kernel
        mbar_expect_tx(&full[i], S::STAGE_BYTES);
        tma_load_2d(base + (size_t)i * S::STAGE_BYTES, &map_w, 0, wrow + i * TILE_M, &full[i]);
      }
      pdl_wait();
      for (int i = 0; i < ahead; ++i)
        tma_load_2d(base + (size_t)i * S::STAGE_BYTES + S::A_BYTES, &map_x, x0 + (kb0 + i) * KB, 0, &full[i]);
      bool ok = true;
      RingCursor c;  // of the stage that block i goes to
      for (int i = 0; i < ahead; ++i) c.next(S::STAGES);
      for (int i = ahead; i < nkb; ++i, c.next(S::STAGES)) {
        ok = mbar_wait(&empty[c.stage], c.parity ^ 1, failed, a.error_flag, 11);
        if (!ok) break;
        mbar_expect_tx(&full[c.stage], S::STAGE_BYTES);
        tma_load_2d(base + (size_t)c.stage * S::STAGE_BYTES, &map_w, 0, wrow + i * TILE_M, &full[c.stage]);
        tma_load_2d(base + (size_t)c.stage * S::STAGE_BYTES + S::A_BYTES, &map_x, x0 + (kb0 + i) * KB, 0, &full[c.stage]);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = umma_idesc_bf16(ROWS, BN);
      bool ok = true;
      RingCursor c;
      for (int i = 0; i < nkb; ++i, c.next(S::STAGES)) {
        ok = mbar_wait(&full[c.stage], c.parity, failed, a.error_flag, 12);
        if (!ok) break;
        tc_fence_after();
        const uint64_t da = umma_desc_sw128(base + (size_t)c.stage * S::STAGE_BYTES);
        const uint64_t db = umma_desc_sw128(base + (size_t)c.stage * S::STAGE_BYTES + S::A_BYTES);
#pragma unroll
        for (int k = 0; k < KB / 16; ++k) umma_bf16_ss(tmem_d, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (i | k) != 0);
        umma_commit(&empty[c.stage]);
      }
      if (ok) umma_commit(d_full);
    }
  } else {
    // Rows of an accumulator of 128 lie in the 128 lanes of tensor memory, those of 64 in the first sixteen of every 32.
    const int r = ROWS == 128 ? (warp & 3) * 32 + lane : (warp & 3) * 16 + lane;
    bool ok = mbar_wait(d_full, 0, failed, a.error_flag, 13);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after();
#pragma unroll 1
      for (int c0 = 0; c0 < BN && c0 < a.m; c0 += 16) {
        float v[16];
        tmem_ld16(tmem_d + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (ROWS == 128 || lane < 16) part[(c0 + j) * ROWS + r] = v[j];
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (splits > 1) {  // every partial sum of the tile is in place
    cluster_arrive();
    cluster_wait();
  }
  pdl_wait();  // nothing may be overwritten before the previous kernel has ended
  if (!*failed) {
    const uint32_t part_addr = smem_u32(part);
    const bool vec = a.ldo % 4 == 0 && a.out_head % 4 == 0 &&  // four results in one store
                     ((out_kind == OUT_F32 ? reinterpret_cast<uintptr_t>(a.out) : reinterpret_cast<uintptr_t>(a.out_h)) & 15) == 0;
    const int pieces = a.m * (ROWS / 4), first = pieces * split / splits, last = pieces * (split + 1) / splits;
    for (int i = first + (int)threadIdx.x; i < last; i += 192) {
      const int j = i / (ROWS / 4), f0 = n0 + (i % (ROWS / 4)) * 4;
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
      if (splits == 1) {
        sum = reinterpret_cast<const float4*>(part)[i];
      } else {
        for (int q = 0; q < splits; ++q) {
          const float4 v = cluster_load4(part_addr + (uint32_t)i * 16u, (uint32_t)q);
          sum.x += v.x;
          sum.y += v.y;
          sum.z += v.z;
          sum.w += v.w;
        }
      }
      const size_t at = (size_t)j * a.ldo + (size_t)head * a.out_head + f0;
      if (vec && f0 + 3 < a.n && (a.act_from <= 0 || f0 + 3 < a.act_from)) {
        if (out_kind == OUT_BF16_ACT) {
          activate_pair(a.act, sum.x, sum.y);
          activate_pair(a.act, sum.z, sum.w);
        }
        if (out_kind == OUT_F32) store4(a.out + at, sum);
        else store4(static_cast<__nv_bfloat16*>(a.out_h) + at, sum);
        continue;
      }
      float y[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int feat = f0 + e;
        if (feat >= a.n) break;
        float v = y[e];
        const bool act_part = a.act_from > 0 && feat >= a.act_from;
        if (out_kind == OUT_BF16_ACT || act_part) {
          float z = 0.f;
          activate_pair(a.act, v, z);
        }
        if (act_part) static_cast<__nv_bfloat16*>(a.out_act)[(size_t)j * a.ldo_act + feat - a.act_from] = __float2bfloat16_rn(v);
        else if (out_kind == OUT_F32) a.out[at + e] = v;
        else static_cast<__nv_bfloat16*>(a.out_h)[at + e] = __float2bfloat16_rn(v);
      }
    }
  }
  if (splits > 1) {  // no block's memory goes away while another reads it
    cluster_arrive();
    cluster_wait();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_d, COLS);
}

// ------------------------------------------------------------------ host side
int sm_count() {
  static const int n = [] {
    int dev = 0, v = 148;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) v = 148;
    return v;
  }();
  return n;
}

// [rows, cols] with row pitch ld, FP32 or BF16, boxes of 32 rows x 128 bytes; false when the layout does not allow it
bool make_out_map(CUtensorMap* map, void* ptr, bool bf16, uint64_t rows, uint64_t cols, uint64_t ld) {
  EncodeTiledFn fn = encode_fn();
  const uint64_t elem = bf16 ? 2 : 4;
  if (!fn || (ld * elem) % 16 != 0 || (reinterpret_cast<uintptr_t>(ptr) & 15)) return false;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * elem};
  cuuint32_t box[2] = {(cuuint32_t)(128 / elem), 32};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, ptr, dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int out_kind_of(const Bf16GemmArgs& a) { return a.out ? OUT_F32 : a.act.kind != ACT_NONE ? OUT_BF16_ACT : OUT_BF16; }

template <int BN>
cudaError_t launch_bn(const Bf16GemmArgs& a, bool pdl, cudaStream_t s) {
  CUtensorMap mx, mw, mo{};
  if (!make_map_bf16(&mx, a.x, a.m, a.k, TILE_M) || !make_map_bf16(&mw, a.w, a.n, a.k, BN)) return cudaErrorInvalidValue;
  const int kind = out_kind_of(a);
  const int tma_out = make_out_map(&mo, kind == OUT_F32 ? (void*)a.out : a.out_h, kind != OUT_F32, a.m, a.n, a.ldo) ? 1 : 0;
  const size_t smem = BfSmem<BN>::BYTES;
  cudaError_t e = cudaFuncSetAttribute(tc_gemm_bf16_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int tiles = ((a.m + TILE_M - 1) / TILE_M) * ((a.n + BN - 1) / BN);
  return launch_kernel(tc_gemm_bf16_kernel<BN>, dim3(std::min(tiles, sm_count())), dim3(192), smem, s, pdl, mx, mw, mo, a, kind, tma_out);
}

template <int BN, int ROWS>
cudaError_t launch_rows_tile(const Bf16GemmArgs& a, int row_tiles, int heads, int splits, bool pdl, cudaStream_t s) {
  CUtensorMap mx, mw;
  if (!make_map_bf16(&mx, a.x, a.m, a.heads ? a.ldx : a.k, BN) || !make_map_bf16(&mw, a.w_tiled, (uint64_t)heads * row_tiles * (a.k / KB) * TILE_M, KB, ROWS))
    return cudaErrorInvalidValue;
  auto kernel = tc_gemm_bf16_rows_kernel<BN, ROWS>;
  const size_t smem = RowsSmem<BN, ROWS>::BYTES;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a.n + ROWS - 1) / ROWS, splits, heads);
  cfg.blockDim = dim3(192);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = splits;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, mx, mw, a, out_kind_of(a));
}

template <int BN>
cudaError_t launch_rows_bn(const Bf16GemmArgs& a, bool pdl, cudaStream_t s) {
  // Parts of k: a power of two that gives every SM at most one block of 128 weight rows, each part of at least two k blocks; eight only
  // where the matrix has eight row tiles or fewer. The parts are where a sum is rounded, and so which way BF16 results behind it fall:
  // other parts were up to 0.4% off in what a model says.
  const int row_tiles = (a.n + TILE_M - 1) / TILE_M, heads = std::max(a.heads, 1), nkb = (a.k + KB - 1) / KB, tiles = row_tiles * heads;
  const int most = tiles <= 8 ? 8 : 4;
  int splits = 1;
  while (splits < most && tiles * splits * 2 <= sm_count() && splits * 4 <= nkb) splits *= 2;
  // Half tiles, the same sums in twice the blocks, where whole ones leave SMs without a second block: steps of 64 sequences of width 2048 with
  // their prompts, 24 of them, Dirurax 26.9 -> 25.5 ms, Sanesun 24.7 -> 23.1 (with four stages instead of six 26.3 and 23.9); 12 sequences of
  // width 1024 the same within the spread.
  return tiles * splits <= sm_count() ? launch_rows_tile<BN, 64>(a, row_tiles, heads, splits, pdl, s)
                                      : launch_rows_tile<BN, 128>(a, row_tiles, heads, splits, pdl, s);
}

}  // namespace

bool gemm_bf16_rows_kernel(int m, int k) { return m <= 64 && k % KB == 0; }

cudaError_t launch_tc_gemm_bf16(const Bf16GemmArgs& a, bool pdl, cudaStream_t s) {
  if (a.m <= 0 || a.n <= 0) return cudaSuccess;
  if (a.heads > 0 && (a.x_head % 8 != 0 || a.ldx % 8 != 0)) return cudaErrorInvalidValue;  // TMA boxes start on 16 bytes
  if ((a.act_from > 0 || a.heads > 0) && (!a.w_tiled || !gemm_bf16_rows_kernel(a.m, a.k))) return cudaErrorInvalidValue;
  if (a.k <= 0 || a.k % 8 != 0 || (!a.out && !a.out_h)) return cudaErrorInvalidValue;
  if (a.w_tiled && a.k % KB == 0) {
    if (a.m <= 16) return launch_rows_bn<16>(a, pdl, s);
    if (a.m <= 32) return launch_rows_bn<32>(a, pdl, s);
    if (a.m <= 64) return launch_rows_bn<64>(a, pdl, s);
  }
  const long long m_tiles = (a.m + TILE_M - 1) / TILE_M;
  if (m_tiles * ((a.n + 255) / 256) >= sm_count()) return launch_bn<256>(a, pdl, s);
  if (m_tiles * ((a.n + 127) / 128) >= 100) return launch_bn<128>(a, pdl, s);
  return launch_bn<64>(a, pdl, s);
}

}  // namespace pg
