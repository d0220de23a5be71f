// One new token per sequence through a recurrent mixer (gated linear attention, delta rules): the cached
// [dim, vdim] FP32 state of every head is read, advanced and written back, with the gates before it and the head norm and
// output gate after it in the same kernel. Everything that enters the recurrence is FP32.
#include <algorithm>
#include <climits>

#include "recurrence.cuh"

namespace pg {
namespace {

// ------------------------------------------------------------------ one token per sequence
// Bound by the state, read and written once, and by the instructions around it. A block takes one head of a sequence after
// another, as many blocks as are resident at a time: while the sums, gates and norms of one state are worked out, the next state
// (into words that the copying thread reads itself) and what goes with it come into shared memory.
// 64 sequences, us (one block per item, loads at the start of each): 16 heads of 64 x 128 26.3 -> 23.3 (2.9 TB/s of state), 32 of
// 64 x 64 34.0 -> 31.6; one sequence, 8 heads of 64 x 128 6.2 -> 4.8.
// The first item's state ahead of the dependency wait, 24 steps of 64 sequences of width 2048 with their prompts: Sanesun 22.8 -> 22.3 ms, Dirurax
// (its attention likewise) 25.1 -> 24.2.
constexpr int STEP_THREADS = 256;

__device__ __forceinline__ void async_copy4(float4* to_shared, const float* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to_shared)), "l"(from) : "memory");
}
__device__ __forceinline__ void async_copy1(float* to_shared, const float* from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(to_shared)), "l"(from) : "memory");
}
__device__ __forceinline__ void async_copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Four neighbouring values as two packed pairs.
struct Quad {
  unsigned long long a, b;
};
__device__ __forceinline__ Quad quad(float4 v) { return Quad{pack2(v.x, v.y), pack2(v.z, v.w)}; }
__device__ __forceinline__ float4 unquad(Quad q) {
  float4 v;
  unpack2(q.a, v.x, v.y);
  unpack2(q.b, v.z, v.w);
  return v;
}
__device__ __forceinline__ Quad fma_quad(float x, Quad y, Quad z) {
  const unsigned long long x2 = pack2(x, x);
  return Quad{fma2(x2, y.a, z.a), fma2(x2, y.b, z.b)};
}

__device__ __host__ inline int pad4(int n) { return (n + 3) & ~3; }
// Floats of one step's inputs in shared memory: key, query, removal rate, value, gate and low-rank columns.
__device__ __host__ inline int step_input_floats(const RecurrenceLayer& l) { return 3 * pad4(l.dim) + 2 * l.dvp + pad4(l.rank); }
inline size_t step_floats(const RecurrenceLayer& l, int buffers) {
  return (size_t)buffers * step_input_floats(l) + 5 * pad4(l.dim) + 2 * l.dvp + std::max(STEP_THREADS, pad4(l.dim)) +
         (size_t)(STEP_THREADS / (l.dvp / 4)) * l.dvp;
}

// An item per block, without the limit on registers that goes with several, or several; STEP_FULL: and every thread owns NR rows
// and four columns of the state, so that nothing is asked per row.
enum { STEP_ONE = 0, STEP_MANY = 1, STEP_FULL = 2 };
constexpr int step_blocks(int nr) { return nr <= 4 ? 4 : nr <= 8 ? 3 : 2; }  // on an SM
// With several items to a block the weights that a thread needs for each of them, all of one head, stay in shared memory, in words that it
// copies and reads itself, where sizes allow (held_at; 0: not). They came from L2 for every item, three round trips of its chain:
// 64 sequences, 16 heads of 64 x 128 20.8 -> 17.6 us, 32 of 64 x 64 29.8 -> 26.0; 24 steps of Dirurax of width 2048 with their prompts
// 23.66 -> 23.13 ms. In registers, for a block's only item, they took 17.37 ms instead of 17.22 (64 steps of one sequence of width 1024: loads in
// front of the dependency wait stand in the way of the product's), and held taps and gates gain the channel rule nothing (21.96 and 21.92).
constexpr int HELD_W = 16, STEP_HELD = HELD_W + 3;  // rows of the decay projection; its bias, bias of the removal rate, norm

template <int NR, int MODE>
__global__ void __launch_bounds__(STEP_THREADS, MODE != STEP_ONE ? step_blocks(NR) : 1) recurrence_step_kernel(RecurrenceStepArgs a, int y_bf16, int ahead_at, int held_at) {
  constexpr bool MANY = MODE != STEP_ONE, FULL = MODE == STEP_FULL;
  extern __shared__ __align__(16) float sm[];
  __shared__ float red[33];
  const RecurrenceLayer& l = a.l;
  const int dk = l.dim, dv = l.vdim, dvp = l.dvp, K = l.heads * dk;
  const int tid = threadIdx.x, head = blockIdx.x % l.heads, seq_step = gridDim.x / l.heads;  // the head of all its items
  const bool delta = l.kind == KIND_DELTA;
  const int dka = pad4(dk), in_floats = step_input_floats(l);  // rows of shared memory start on 16-byte boundaries
  float4* rp = reinterpret_cast<float4*>(sm + (MANY ? 2 : 1) * in_floats);  // [dk] of a row of the state: decay, key, query, a * u
  float* us = reinterpret_cast<float*>(rp + dka);  // [dk] unit key
  float* ds = us + dka;            // [dvp] u^T S
  float* os = ds + dvp;            // [dvp]
  float* zs = os + dvp;            // [max(256, dk)] partial sums of the decay projection
  float* part = zs + (dk > STEP_THREADS ? dka : STEP_THREADS);  // [KG][dvp]
  const int dv4 = dvp / 4, KG = STEP_THREADS / dv4;
  const int c4 = tid % dv4, kg = tid / dv4;
  const bool active = FULL || kg < KG;
  const int own = FULL ? INT_MAX : dk;  // rows below are there
  float4* ahead = reinterpret_cast<float4*>(sm + ahead_at) + tid;  // [NR][STEP_THREADS], this thread's column
  auto fetch = [&](int seq, float* in) {
    const float* p = a.p + (size_t)seq * a.ldp;
    for (int c = tid; c < dk; c += STEP_THREADS) {
      async_copy1(in + c, p + l.off_k + head * dk + c);
      async_copy1(in + dka + c, p + l.off_q + head * dk + c);
      if (delta) async_copy1(in + 2 * dka + c, p + l.off_a + head * dk + c);
    }
    for (int c = tid; c < dv; c += STEP_THREADS) {
      async_copy1(in + 3 * dka + c, p + l.off_v + head * dv + c);
      async_copy1(in + 3 * dka + dvp + c, p + l.off_g + head * dv + c);
    }
    for (int r = tid; r < l.rank; r += STEP_THREADS) async_copy1(in + 3 * dka + 2 * dvp + r, p + l.off_t + r);
  };

  for (int c = dv + tid; c < dvp; c += STEP_THREADS) {  // padding of the value rows
    sm[3 * dka + c] = 0.f;
    if (MANY) sm[in_floats + 3 * dka + c] = 0.f;
  }
  grid_dep_launch();
  // States, convolution inputs and positions were written before this step began, and a step's first launch waits for all that is before it:
  // the first item's are asked for while the kernel in front is still running.
  const int first = blockIdx.x / l.heads;
  bool fresh = a.pos[first] == 0;
  constexpr int NRR = NR > 0 ? NR : 1;
  Quad st[NRR];
#pragma unroll
  for (int i = 0; i < NRR; ++i) st[i] = Quad{0, 0};
  if (NR > 0 && active && !fresh) {
    const float* from = a.state + ((size_t)first * l.heads + head) * dk * dvp + (size_t)kg * dvp + c4 * 4;
#pragma unroll
    for (int i = 0; i < NRR; ++i)
      if (kg + i * KG < own) st[i] = quad(load4(from + (size_t)i * KG * dvp));
  }
  const bool hold = MANY && held_at > 0;
  float* held = sm + held_at + tid;
  if (hold) {
    const int RG = STEP_THREADS / dk;  // as below
    if (tid < RG * dk)
      for (int r = tid / dk, at = 0; r < l.rank; r += RG, at += STEP_THREADS) async_copy1(held + at, l.w2 + (size_t)r * K + head * dk + tid % dk);
    if (tid < dk) async_copy1(held + HELD_W * STEP_THREADS, l.b2 + head * dk + tid);
    if (tid < dk && delta) async_copy1(held + (HELD_W + 1) * STEP_THREADS, l.a_bias + head * dk + tid);
    if (tid < dv) async_copy1(held + (HELD_W + 2) * STEP_THREADS, l.norm + (delta ? head * dv : 0) + tid);
  }
  grid_dep_wait();
  fetch(first, sm);
  int flip = 0;
  for (int seq = first; seq < a.batch; seq += seq_step, flip ^= 1) {
    const int next = MANY ? seq + seq_step : a.batch;
    const float *ks = sm + flip * in_floats, *qs = ks + dka, *as = qs + dka, *vs = as + dka, *gs = vs + dvp;
    float* ts = sm + flip * in_floats + 3 * dka + 2 * dvp;
    float* S = a.state + ((size_t)seq * l.heads + head) * dk * dvp + (size_t)kg * dvp + c4 * 4;  // this thread's first row
    const size_t pitch = (size_t)KG * dvp;
    const bool stored = active && !fresh;
    async_copies_done();
    if (NR > 0 && MANY && seq != first) {
#pragma unroll
      for (int i = 0; i < NRR; ++i) st[i] = stored && kg + i * KG < own ? quad(ahead[i * STEP_THREADS]) : Quad{0, 0};
    }
    if (delta)
      for (int r = tid; r < l.rank; r += STEP_THREADS) ts[r] = tanhf(ts[r]);  // this thread's copies
    float kk = 0.f;
    for (int c = tid; c < dk; c += STEP_THREADS) kk += ks[c] * ks[c];
    kk = block_sum(kk, red);  // also orders the copies, and the last item's reads of the other buffer before the next ones
    if (next < a.batch) {
      fetch(next, sm + (flip ^ 1) * in_floats);
      if (NR > 0 && active) {
        const float* from = S + (size_t)seq_step * l.heads * dk * dvp;
#pragma unroll
        for (int i = 0; i < NRR; ++i)
          if (kg + i * KG < own) async_copy4(ahead + i * STEP_THREADS, from + i * pitch);
      }
    }
    const int next_pos = next < a.batch ? a.pos[next] : 0;
    const float inv_norm = 1.f / sqrtf(kk + UNIT_EPS);
    // second half of the decay projection: RG threads share a channel, so that its weights arrive in one round trip or two
    const int RG = dk >= STEP_THREADS ? 1 : STEP_THREADS / dk;
    if (hold) {
      if (tid < RG * dk) {
        float z = 0.f;
#pragma unroll 8
        for (int r = tid / dk, at = 0; r < l.rank; r += RG, at += STEP_THREADS) z = fmaf(held[at], ts[r], z);
        zs[tid] = z;
      }
    } else {
      for (int i = tid; i < RG * dk; i += STEP_THREADS) {
        const int c = i % dk, g = i / dk;
        const float* __restrict__ w2 = l.w2 + head * dk + c;
        float z = 0.f;
#pragma unroll 16
        for (int r = g; r < l.rank; r += RG) z = fmaf(w2[(size_t)r * K], ts[r], z);
        zs[i] = z;
      }
    }
    __syncthreads();
    for (int c = tid; c < dk; c += STEP_THREADS) {
      const int ch = head * dk + c;
      float z = hold ? held[HELD_W * STEP_THREADS] : l.b2[ch];
      for (int g = 0; g < RG; ++g) z += zs[g * dk + c];
      float b = 0.f;
      if (delta) {
        const float u = ks[c] * inv_norm;
        us[c] = u;
        b = sigmoid_f(as[c] + (hold ? held[(HELD_W + 1) * STEP_THREADS] : l.a_bias[ch])) * u;
      }
      rp[c] = make_float4(decay_of(l.kind, z, l.inv_tau), ks[c], qs[c], b);
    }
    __syncthreads();
    const int count = NR > 0 ? NRR : (dk + KG - 1) / KG;
    if (delta) {
      Quad d = {0, 0};
      if (stored) {
#pragma unroll
        for (int i = 0; i < count; ++i) {
          const int r = kg + i * KG;
          if (r >= own) break;
          d = fma_quad(us[r], NR > 0 ? st[NR > 0 ? i : 0] : quad(load4(S + i * pitch)), d);
        }
      }
      if (active) store4(part + (size_t)kg * dvp + c4 * 4, unquad(d));
      __syncthreads();
      for (int c = tid; c < dvp; c += STEP_THREADS) {
        float sum = 0.f;
#pragma unroll 8
        for (int g = 0; g < KG; ++g) sum += part[(size_t)g * dvp + c];
        ds[c] = sum;
      }
      __syncthreads();
    }
    if (active) {
      const Quad v = quad(load4(vs + c4 * 4)), d = delta ? quad(load4(ds + c4 * 4)) : Quad{0, 0}, zero = {0, 0};
      Quad o = {0, 0};
#pragma unroll
      for (int i = 0; i < count; ++i) {
        const int r = kg + i * KG;
        if (r >= own) break;
        const float4 row = rp[r];
        Quad x = NR > 0 ? st[NR > 0 ? i : 0] : fresh ? Quad{0, 0} : quad(load4(S + i * pitch));
        x = fma_quad(row.x, x, fma_quad(row.y, v, delta ? fma_quad(-row.w, d, zero) : zero));
        store4(S + i * pitch, unquad(x));
        o = fma_quad(row.z, x, o);
      }
      store4(part + (size_t)kg * dvp + c4 * 4, unquad(o));
    }
    __syncthreads();
    float sq = 0.f;
    for (int c = tid; c < dv; c += STEP_THREADS) {
      float sum = 0.f;
#pragma unroll 8
      for (int g = 0; g < KG; ++g) sum += part[(size_t)g * dvp + c];
      sum *= l.q_scale;
      os[c] = sum;
      sq += sum * sum;
    }
    sq = block_sum(sq, red);
    const float rinv = 1.f / sqrtf(sq / (float)dv + l.eps);
    for (int c = tid; c < dv; c += STEP_THREADS) {
      const float gate = delta ? sigmoid_f(gs[c]) : silu_f(gs[c]);
      const float y = os[c] * rinv * (hold ? held[(HELD_W + 2) * STEP_THREADS] : l.norm[delta ? head * dv + c : c]) * gate * l.out_scale;
      const size_t at = (size_t)seq * a.ldy + head * dv + c;
      if (y_bf16) static_cast<__nv_bfloat16*>(a.y)[at] = __float2bfloat16_rn(y);
      else static_cast<float*>(a.y)[at] = y;
    }
    fresh = next_pos == 0;
  }
}

// ------------------------------------------------------------------ channel delta rule
// Block = one head of a sequence, then of another, as in recurrence_step_kernel. A thread owns four columns of NR rows of the
// state (NR = 0: it is read twice instead). The unit lengths of k and q are factors of sums, so that the rows go on as they leave
// the convolutions.
// 64 sequences, 16 heads of 128 x 128: 46 -> 41 us (3.2 TB/s; DRAM 22% busy and half of the issue slots taken in the former kernel).
constexpr int CH_THREADS = 512, CH_WARPS = CH_THREADS / 32;

// Floats of one step's inputs in shared memory: `taps` rows of key, query and value inputs, decay and gate columns, write strength.
__device__ __host__ inline int channel_input_floats(const RecurrenceLayer& l) { return l.taps * (2 * l.dim + l.vdim) + l.dim + l.vdim + 1; }
inline size_t channel_floats(const RecurrenceLayer& l, int buffers) {
  return 4 * (size_t)pad4(l.dim) + l.dvp + (size_t)(CH_THREADS / (l.dvp / 4)) * l.dvp + (size_t)buffers * channel_input_floats(l);
}
constexpr int channel_blocks(int nr) { return nr > 0 && nr <= 8 ? 2 : 1; }

template <int NR, int MODE>
__global__ void __launch_bounds__(CH_THREADS, channel_blocks(NR)) channel_step_kernel(RecurrenceStepArgs a, int y_bf16, int ahead_at, int) {
  constexpr bool MANY = MODE != STEP_ONE, FULL = MODE == STEP_FULL;
  extern __shared__ __align__(16) float sm[];
  __shared__ float red[CH_WARPS], lengths[3];  // of key and query; write strength
  const RecurrenceLayer& l = a.l;
  const int dk = l.dim, dv = l.vdim, dvp = l.dvp, dka = pad4(dk), rep = l.heads / l.kv_heads;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, head = blockIdx.x % l.heads, seq_step = gridDim.x / l.heads, kv = head / rep;
  const int dv4 = dvp / 4, KG = CH_THREADS / dv4, c4 = tid % dv4, kg = tid / dv4;
  const bool active = FULL || kg < KG;
  const int own = FULL ? INT_MAX : dk;   // rows below are there
  float* rp = sm;                        // [dk][4] of a row of the state: decay, key, query, unused
  float* vs = rp + 4 * dka;              // [dvp] value, then what is written
  float* part = vs + dvp;                // [KG][dvp]
  float* inputs = part + (size_t)KG * dvp;
  const int rows = 2 * dk + dv, in_floats = channel_input_floats(l);
  float4* ahead = reinterpret_cast<float4*>(sm + ahead_at) + tid;  // [NR][CH_THREADS], this thread's column
  // column j of an input row: key, query, value
  auto column = [&](int j) { return j < dk ? l.off_k + kv * dk + j : j < 2 * dk ? l.off_q + kv * dk + j - dk : l.off_v + head * dv + j - 2 * dk; };
  auto fetch_past = [&](int seq, int slot, float* in) {
    const float* taps = a.taps + (size_t)seq * l.taps * l.channels;
    for (int j = tid; j < rows; j += CH_THREADS) {
      const float* past = taps + (size_t)slot * l.channels + column(j) - l.off_q;
      for (int back = 1, at = slot; back < l.taps; ++back) {
        past += at == 0 ? (l.taps - 1) * l.channels : -l.channels;
        at = at == 0 ? l.taps - 1 : at - 1;
        async_copy1(in + back * rows + j, past);
      }
    }
  };
  auto fetch_now = [&](int seq, float* in) {
    const float *p = a.p + (size_t)seq * a.ldp, *z = a.z + (size_t)seq * a.ldz;
    for (int j = tid; j < rows; j += CH_THREADS) async_copy1(in + j, p + column(j));
    in += l.taps * rows;
    for (int j = tid; j < dk + dv + 1; j += CH_THREADS)
      async_copy1(in + j, j < dk ? z + head * dk + j : j < dk + dv ? z + l.heads * dk + head * dv + j - dk : p + l.off_b + head);
  };

  grid_dep_launch();
  const int first = blockIdx.x / l.heads;  // before the dependency wait: as in recurrence_step_kernel
  int pos = a.pos[first], slot = pos % l.taps, flip = 0;
  fetch_past(first, slot, inputs);
  constexpr int NRR = NR > 0 ? NR : 1;
  Quad st[NRR];
#pragma unroll
  for (int i = 0; i < NRR; ++i) st[i] = Quad{0, 0};
  if (NR > 0 && active && pos != 0) {
    const float* from = a.state + ((size_t)first * l.heads + head) * dk * dvp + (size_t)kg * dvp + c4 * 4;
#pragma unroll
    for (int i = 0; i < NRR; ++i)
      if (kg + i * KG < own) st[i] = quad(load4(from + (size_t)i * KG * dvp));
  }
  grid_dep_wait();
  fetch_now(first, inputs);
  int next_pos = MANY && first + seq_step < a.batch ? a.pos[first + seq_step] : 0;
  for (int seq = first; seq < a.batch; seq += seq_step, flip ^= 1) {
    const int next = MANY ? seq + seq_step : a.batch;
    const float *in = inputs + flip * in_floats, *zs = in + l.taps * rows;  // [dk] decay, [dv] gate, write strength
    float* S = a.state + ((size_t)seq * l.heads + head) * dk * dvp + (size_t)kg * dvp + c4 * 4;  // this thread's first row
    const size_t pitch = (size_t)KG * dvp;
    const bool fresh = pos == 0, stored = active && !fresh;
    async_copies_done();
    if (NR > 0 && MANY && seq != first) {
#pragma unroll
      for (int i = 0; i < NRR; ++i) st[i] = stored && kg + i * KG < own ? quad(ahead[i * CH_THREADS]) : Quad{0, 0};
    }
    float* taps = a.taps + ((size_t)seq * l.taps + slot) * l.channels;
    for (int c = dv + tid; c < dvp; c += CH_THREADS) vs[c] = 0.f;
    for (int j = tid; j < rows; j += CH_THREADS) {  // this thread's copies
      const int ch = column(j) - l.off_q;
      const float now = in[j];
      float x = 0.f;
      for (int back = l.taps - 1; back > 0; --back)
        if (pos >= back) x = fmaf(l.conv[(size_t)(l.taps - 1 - back) * l.channels + ch], in[back * rows + j], x);
      x = silu_f(fmaf(l.conv[(size_t)(l.taps - 1) * l.channels + ch], now, x));
      (j < dk ? rp + 4 * j + 1 : j < 2 * dk ? rp + 4 * (j - dk) + 2 : vs + j - 2 * dk)[0] = x;
      // the input is cached where no token that still matters lies; one block per group caches the shared q and k
      if (head % rep == 0 || j >= 2 * dk) taps[ch] = now;
    }
    __syncthreads();  // also the copies of the other threads, and the last item's reads of the other buffer before the next ones
    pos = next_pos;
    slot = pos % l.taps;
    if (next < a.batch) {
      fetch_past(next, slot, inputs + (flip ^ 1) * in_floats);
      fetch_now(next, inputs + (flip ^ 1) * in_floats);
      if (NR > 0 && active) {
        const float* from = S + (size_t)seq_step * l.heads * dk * dvp;
#pragma unroll
        for (int i = 0; i < NRR; ++i)
          if (kg + i * KG < own) async_copy4(ahead + i * CH_THREADS, from + i * pitch);
      }
      next_pos = next + seq_step < a.batch ? a.pos[next + seq_step] : 0;
    }
    for (int c = tid; c < dk; c += CH_THREADS) rp[4 * c] = channel_decay(l, head, head * dk + c, zs[c]);
    if (warp >= CH_WARPS - 2) {  // squared lengths
      const int at = warp == CH_WARPS - 1 ? 2 : 1;
      float sum = 0.f;
      for (int c = lane; c < dk; c += 32) sum += rp[4 * c + at] * rp[4 * c + at];
      sum = lane_sum(sum);
      if (lane == 0) lengths[at - 1] = 1.f / sqrtf(sum + UNIT_EPS);
    } else if (warp == CH_WARPS - 3 && lane == 0) {
      lengths[2] = sigmoid_f(zs[dk + dv]);
    }
    __syncthreads();
    const int count = NR > 0 ? NRR : (dk + KG - 1) / KG;
    const float4* rows4 = reinterpret_cast<const float4*>(rp);
    if (active) {
      Quad d = {0, 0};
      if (stored) {
#pragma unroll
        for (int i = 0; i < count; ++i) {
          const int r = kg + i * KG;
          if (r >= own) break;
          const float4 row = rows4[r];
          d = fma_quad(row.x * row.y, NR > 0 ? st[NR > 0 ? i : 0] : quad(load4(S + i * pitch)), d);
        }
      }
      store4(part + (size_t)kg * dvp + c4 * 4, unquad(d));
    }
    __syncthreads();
    const float ki = lengths[0], qi = lengths[1], beta = lengths[2];
    for (int c = tid; c < dvp; c += CH_THREADS) {
      float sum = 0.f;
#pragma unroll 8
      for (int g = 0; g < KG; ++g) sum += part[(size_t)g * dvp + c];
      vs[c] = beta * ki * (vs[c] - ki * sum);
    }
    __syncthreads();
    if (active) {
      const Quad v = quad(load4(vs + c4 * 4)), zero = {0, 0};
      Quad o = {0, 0};
#pragma unroll
      for (int i = 0; i < count; ++i) {
        const int r = kg + i * KG;
        if (r >= own) break;
        const float4 row = rows4[r];
        Quad x = NR > 0 ? st[NR > 0 ? i : 0] : fresh ? Quad{0, 0} : quad(load4(S + i * pitch));
        x = fma_quad(row.x, x, fma_quad(row.y, v, zero));
        store4(S + i * pitch, unquad(x));
        o = fma_quad(row.z, x, o);
      }
      store4(part + (size_t)kg * dvp + c4 * 4, unquad(o));
    }
    __syncthreads();
    float out = 0.f;  // one column per thread: dv <= CH_THREADS
    if (tid < dv) {
#pragma unroll 8
      for (int g = 0; g < KG; ++g) out += part[(size_t)g * dvp + tid];
      out *= qi * l.q_scale;
    }
    const float sq = lane_sum(out * out);
    if (lane == 0) red[warp] = sq;
    __syncthreads();
    if (tid < dv) {
      float total = 0.f;
#pragma unroll
      for (int i = 0; i < CH_WARPS; ++i) total += red[i];
      const float y = out / sqrtf(total / (float)dv + l.eps) * l.norm[tid] * sigmoid_f(zs[dk + tid]) * l.out_scale;
      const size_t at = (size_t)seq * a.ldy + head * dv + tid;
      if (y_bf16) static_cast<__nv_bfloat16*>(a.y)[at] = __float2bfloat16_rn(y);
      else static_cast<float*>(a.y)[at] = y;
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

// Shared memory of a block where `per_sm` of them share an SM (of 228 KB, 1 KB of it taken with every block).
constexpr size_t step_smem_limit(int per_sm) { return (size_t)227 * 1024 / per_sm - 1024; }

// The instances that hold NR rows of the state per thread.
typedef void (*StepKernel)(RecurrenceStepArgs, int, int, int);
struct StepKernels {
  StepKernel one, some, full;
  int nr, threads, per_sm;
};
template <int NR>
StepKernels channel_kernels() {
  constexpr int SOME = NR == 0 ? STEP_ONE : STEP_MANY, FULL = NR == 0 ? STEP_ONE : STEP_FULL;
  return {channel_step_kernel<NR, STEP_ONE>, channel_step_kernel<NR, SOME>, channel_step_kernel<NR, FULL>, NR, CH_THREADS, channel_blocks(NR)};
}
template <int NR>
StepKernels gated_kernels() {
  constexpr int SOME = NR == 0 ? STEP_ONE : STEP_MANY, FULL = NR == 0 ? STEP_ONE : STEP_FULL;
  return {recurrence_step_kernel<NR, STEP_ONE>, recurrence_step_kernel<NR, SOME>, recurrence_step_kernel<NR, FULL>, NR, STEP_THREADS, step_blocks(NR)};
}

// As many blocks as are resident at `per_sm` an SM, where there are more items than that and the kernel keeps the state in
// registers (nr > 0): a multiple of the heads then, since a block stays with one head. Else a block per item. Whole steps, us, a block
// per item and several, from the first number of sequences past residency on: Dirurax of width 2048 (592 blocks of the delta rule, 432 of
// the gated one) 19 627 / 607, 27 663 / 632, 28 689 / 602, 64 966 / 795; of width 1024 38 466 / 446, 64 550 / 465; Sanesun of width
// 2048 (288 blocks) 19 572 / 557, 32 592 / 587, 37 629 / 644, 64 750 / 732.
cudaError_t launch_step(const StepKernels& k, const RecurrenceStepArgs& a, int yb, bool pdl, cudaStream_t s) {
  const RecurrenceLayer& l = a.l;
  auto floats = [&](int buffers) { return l.kind == KIND_CHANNEL ? channel_floats(l, buffers) : step_floats(l, buffers); };
  const int items = l.heads * a.batch, resident = k.per_sm * sm_count() / l.heads * l.heads;
  const size_t smem = floats(1) * sizeof(float), ahead = (floats(2) + 3) / 4 * 16, bytes = ahead + (size_t)k.nr * k.threads * 16;
  if (k.nr == 0 || resident == 0 || items <= resident || bytes > step_smem_limit(k.per_sm))
    return launch_kernel(k.one, dim3(items), dim3(k.threads), smem, s, pdl, a, yb, 0, 0);
  const bool fits = l.kind != KIND_CHANNEL && l.dim <= STEP_THREADS && l.vdim <= STEP_THREADS && l.rank <= HELD_W * (STEP_THREADS / l.dim);
  const size_t held = (size_t)STEP_HELD * STEP_THREADS * sizeof(float);
  const bool hold = fits && bytes + held <= step_smem_limit(k.per_sm);
  const bool full = l.dim == k.nr * (k.threads / (l.dvp / 4)) && k.threads % (l.dvp / 4) == 0;
  return launch_kernel(full ? k.full : k.some, dim3(resident), dim3(k.threads), bytes + (hold ? held : 0), s, pdl, a, yb, (int)(ahead / sizeof(float)),
                       hold ? (int)(bytes / sizeof(float)) : 0);
}

cudaError_t launch_channel_step(const RecurrenceStepArgs& a, int yb, bool pdl, cudaStream_t s) {
  const RecurrenceLayer& l = a.l;
  const int kg = CH_THREADS / (l.dvp / 4), nr = (l.dim + kg - 1) / kg;
  if (l.dvp > CH_THREADS) return cudaErrorInvalidValue;
  if (nr <= 2) return launch_step(channel_kernels<2>(), a, yb, pdl, s);
  if (nr <= 4) return launch_step(channel_kernels<4>(), a, yb, pdl, s);
  if (nr <= 8) return launch_step(channel_kernels<8>(), a, yb, pdl, s);
  if (nr <= 16) return launch_step(channel_kernels<16>(), a, yb, pdl, s);
  return launch_step(channel_kernels<0>(), a, yb, pdl, s);
}

}  // namespace

// The limits on shared memory belong to the kernels, which layers, models and threads share: they are set once, to the most that a
// layer of any size asks for.
cudaError_t init_recurrence_step_attributes() {
  for (const StepKernels& k : {channel_kernels<2>(), channel_kernels<4>(), channel_kernels<8>(), channel_kernels<16>(), channel_kernels<0>(),
                               gated_kernels<4>(), gated_kernels<8>(), gated_kernels<16>(), gated_kernels<0>()}) {
    cudaError_t e = cudaFuncSetAttribute(k.one, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)step_smem_limit(1));
    if (e == cudaSuccess && k.nr > 0) e = cudaFuncSetAttribute(k.some, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)step_smem_limit(k.per_sm));
    if (e == cudaSuccess && k.nr > 0) e = cudaFuncSetAttribute(k.full, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)step_smem_limit(k.per_sm));
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

size_t recurrence_state_floats(const RecurrenceLayer& l) { return (size_t)l.heads * l.dim * l.dvp; }

cudaError_t launch_recurrence_step(const RecurrenceStepArgs& a, bool y_bf16, bool pdl, cudaStream_t s) {
  const RecurrenceLayer& l = a.l;
  if (l.kind == KIND_CHANNEL) return launch_channel_step(a, y_bf16 ? 1 : 0, pdl, s);
  const int dv4 = l.dvp / 4, kg = STEP_THREADS / dv4, nr = (l.dim + kg - 1) / kg;
  if (dv4 > STEP_THREADS) return cudaErrorInvalidValue;
  const int yb = y_bf16 ? 1 : 0;
  if (nr <= 4) return launch_step(gated_kernels<4>(), a, yb, pdl, s);
  if (nr <= 8) return launch_step(gated_kernels<8>(), a, yb, pdl, s);
  if (nr <= 16) return launch_step(gated_kernels<16>(), a, yb, pdl, s);
  return launch_step(gated_kernels<0>(), a, yb, pdl, s);
}

}  // namespace pg
