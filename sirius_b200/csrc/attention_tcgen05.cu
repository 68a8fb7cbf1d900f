// Attention with 64-channel heads on the sm_100a tensor cores, without the S x S matrices in memory.
//
//   attention_fwd_kernel<CAUSAL>   out = softmax(Q K^T * scale) V; the maximum and the inverse sum of every row are kept
//   attention_bwd_kernel<KV>       causal; KV = false: dQ of 128 queries and the row terms dot = sum P dP,
//                                  KV = true: dK and dV of 128 keys
//
// Heads are addressed in place inside the fused projection through 4-D tensor maps (channel, position, head, batch).
// Every product is a tcgen05.mma over 128 x 64 bf16 tiles that TMA lays out with the 128-byte swizzle; a tile with
// one position per 128-byte row serves as a K-major operand (reduction over channels) and, through another
// descriptor, as an MN-major one (reduction over positions), so nothing is ever transposed.
//
// The arithmetic is that of the score-matrix path (batched GEMM, softmax pass, batched GEMM, which other head sizes
// take) to the last bit: scores and dP are rounded to bf16, the row sums add the same elements in the same order (32
// interleaved partial sums per row, combined as a warp's butterfly does), probabilities are normalised before they are
// rounded, the tensor-core reductions run over the same 16-element steps in the same order. A deep network turns any
// other rounding of one layer into another gradient (2 to 3 % in the 2-norm after 24 layers), so this is what keeps runs,
// and heads of other sizes, comparable. The price is that a row's maximum and sum are known before its
// probabilities are formed: the forward kernel walks the keys three times (maximum, sum, output), the dQ kernel twice
// (dot, output). Recomputing a tile costs 512 tensor-core clocks or less; reading and writing it as bf16 took more.
//
// What bounds it: the arithmetic per score. One exponential (16 a clock and SM: 1024 clocks per 128 x 128 tile) and, in
// the backward kernels, about 9 instructions per element at 128 lanes a clock, against 256 to 512 clocks for the
// products of a tile; memory traffic is Q, K, V, O and their gradients once, the repeats come out of L2.
// The score-matrix path moved 10 to 14 S x S matrices per layer through HBM.
// Measured, 8 sequences of 1024, 12 heads: forward 61 us, backward 153 us, where the score-matrix path took 740 us for
// both (GEMMs 276, softmax 166, transposes 298); 4 x 2048 with 14 query and 2 KV heads: 109 and 271 us against 1650 us.
// (Longest rows first within a head only, instead of over the whole grid: 81, 199, 157 and 377 us; masks in every tile
// instead of the tiles on the edge: 65, 179, 122 and 331 us.)
// Two compute warps per scheduler (a thread with all 128 columns of a row) took 140 and 249 us: the chain of a tile
// (product, wait, load, arithmetic, store) then leaves schedulers idle.
//
// Every sum has a fixed order: dK/dV and dQ come from two launches that each recompute the scores, instead of one
// with floating-point atomics on dQ, so a step repeats bit for bit.
#include <cuda.h>

#include "common.cuh"
#include "ops.cuh"
#include "ptx.cuh"

namespace srt {

int* tc_status_device_ptr();  // igemm_tcgen05.cu
// igemm_tcgen05.cu: tensor map of a batched bf16 operand (channel, row, z1, z2), boxes of 64 channels x box_rows
int tmap_batched_bf16(CUtensorMap* tm, const void* base, uint64_t kdim, uint64_t rows, uint64_t z1, uint64_t z2, uint64_t ld,
                      uint64_t s1, uint64_t s2, uint32_t box_rows);

namespace {

using namespace ptx;
using bf16 = __nv_bfloat16;

constexpr int HD = 64;                 // channels of a head
constexpr int TR = 128;                // positions of a tile
constexpr int TILE_BYTES = TR * HD * 2;
constexpr int SLAB_BYTES = TR * 128;   // 128 rows x 64 bf16, 128-byte swizzle
enum { W_ATT_LOAD = 0x21, W_ATT_MMA = 0x22, W_ATT_COMPUTE = 0x23 };

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
// Pairs of fp32 values in one 64-bit register: the packed add and multiply round each half as the scalar ones do.
__device__ __forceinline__ uint64_t pair(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ uint64_t pair(float lo, float hi) { return pair(__float_as_uint(lo), __float_as_uint(hi)); }
__device__ __forceinline__ void split(uint64_t v, float& lo, float& hi) {
  uint32_t a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v));
  lo = __uint_as_float(a);
  hi = __uint_as_float(b);
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint32_t round2(uint64_t v) {  // to a pair of bf16
  float lo, hi;
  split(v, lo, hi);
  return pack2(lo, hi);
}
__device__ __forceinline__ uint64_t widen2(uint32_t w) { return pair(w << 16, w & 0xffff0000u); }
// exp(bf16(s * scale) - max) of two scores, as 2^(x log2 e); results below 2^-126 become zero
__device__ __forceinline__ uint64_t exp2x(uint32_t s0, uint32_t s1, uint64_t scale, uint64_t neg_max) {
  const uint64_t log2e = pair(1.4426950408889634f, 1.4426950408889634f);
  float a, b;
  split(mul2(add2(widen2(round2(mul2(pair(s0, s1), scale))), neg_max), log2e), a, b);
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(a));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(b));
  return pair(a, b);
}
// Scores of columns beyond `last` (before `first`) become -inf, whose exponential is exactly zero. Only the blocks on the edge
// call these: masks inside the loops over the columns cost every block a compare and a select per element.
__device__ __forceinline__ void hide(uint32_t (&s)[32], int last) {
#pragma unroll
  for (int c = 0; c < 32; ++c)
    if (c > last) s[c] = 0xff800000u;
}
__device__ __forceinline__ void hide_before(uint32_t (&s)[32], int first) {
#pragma unroll
  for (int c = 0; c < 32; ++c)
    if (c < first) s[c] = 0xff800000u;
}
// The bounded wait of the compute warps, one outcome for the whole warp. They poll without sleeping: nothing else runs on
// their schedulers meanwhile but each other, and a sleep would add to the serial chain of a tile.
__device__ __forceinline__ bool wait_all(uint32_t bar, uint32_t parity, int* status, int code) {
  bool ok = mbar_try_wait(bar, parity);
  if (!ok) {
    const long long t0 = clock64();
    while (!(ok = mbar_try_wait(bar, parity)))
      if (clock64() - t0 > kWaitLimitCycles) {
        atomicCAS(status, 0, code);
        break;
      }
  }
  return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ void warp_arrive(uint32_t bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}
// 128 x 128 (two K-major 128 x 64 operands) and 128 x 64 += [128 x 128 K-major, two slabs] x [128 positions x 64
// MN-major]; issued by one thread.
__device__ __forceinline__ void mma_scores(uint32_t d, uint32_t a, uint32_t b) {
  constexpr uint32_t idesc = make_idesc_bf16(TR, TR, 0, 0);
#pragma unroll
  for (int k = 0; k < HD / 16; ++k)
    umma_bf16(d, make_smem_desc_sw128(a + k * 32, 0, 1024), make_smem_desc_sw128(b + k * 32, 0, 1024), idesc, k != 0 ? 1u : 0u);
}
__device__ __forceinline__ void mma_accumulate(uint32_t d, uint32_t a, uint32_t b, bool first) {
  constexpr uint32_t idesc = make_idesc_bf16(TR, HD, 0, 1);
#pragma unroll
  for (int k = 0; k < TR / 16; ++k)
    umma_bf16(d, make_smem_desc_sw128(a + (k >> 2) * SLAB_BYTES + (k & 3) * 32, 0, 1024),
              make_smem_desc_sw128(b + k * 2048, 8192, 1024), idesc, (!first || k != 0) ? 1u : 0u);
}
// 32 fp32 tensor-memory columns of this thread's lane, scaled, rounded and stored as 64 bytes of an output row.
__device__ __forceinline__ void store_half_row(uint32_t taddr, float scale, bf16* out, bool live) {
  uint32_t acc[32];
  tmem_ld_32x32b_x32(taddr, acc);
  tmem_ld_wait();
  if (!live) return;
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    uint4 o;
    o.x = pack2(__uint_as_float(acc[v * 8 + 0]) * scale, __uint_as_float(acc[v * 8 + 1]) * scale);
    o.y = pack2(__uint_as_float(acc[v * 8 + 2]) * scale, __uint_as_float(acc[v * 8 + 3]) * scale);
    o.z = pack2(__uint_as_float(acc[v * 8 + 4]) * scale, __uint_as_float(acc[v * 8 + 5]) * scale);
    o.w = pack2(__uint_as_float(acc[v * 8 + 6]) * scale, __uint_as_float(acc[v * 8 + 7]) * scale);
    *reinterpret_cast<uint4*>(out + v * 8) = o;
  }
}

// ---- forward ------------------------------------------------------------------------------------------
// One CTA: 128 queries of one head. Warps 0-7 softmax (warps w and w + 4 share the rows of a tensor-memory lane quarter, 64
// columns of every tile each), warp 8 TMA, warp 9 MMA and tensor memory (columns 0-127 scores, 128-191 output). The score
// product of the next tile is issued as soon as the current one has been read into registers, so it runs beside the
// arithmetic; two CTAs share an SM (97 KB of shared memory, 256 tensor-memory columns each), one's waits hide behind
// the other's arithmetic.
constexpr int FWD_THREADS = 320;
constexpr int FWD_NS = 3;  // ring of K and V tiles in the order the MMAs read them
constexpr size_t fwd_smem_bytes() { return 1024 + (size_t)TILE_BYTES * (1 + FWD_NS) + 2 * SLAB_BYTES + 128; }

struct AttFwdParams {
  bf16* O;
  float *row_max, *row_inv;  // [B*H][s_pad], or null; the maximum is stored negated
  int S, s_pad, H, kv_div;
  long long ldo, o_s1, o_s2;
  float scale;
  int* status;
};

template <bool CAUSAL>
__global__ void __launch_bounds__(FWD_THREADS, 2)
attention_fwd_kernel(const AttFwdParams p, const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                     const __grid_constant__ CUtensorMap tv) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sQ = smem_u32(base), sKV = sQ + TILE_BYTES, sP = sKV + FWD_NS * TILE_BYTES;
  uint64_t* bars = (uint64_t*)(base + TILE_BYTES * (1 + FWD_NS) + 2 * SLAB_BYTES);
  const uint32_t q_full = smem_u32(bars), kv_full = q_full + 8, kv_empty = kv_full + 8 * FWD_NS,
                 s_full = kv_empty + 8 * FWD_NS, s_free = s_full + 8, p_ready = s_free + 8, o_done = p_ready + 8;
  uint32_t* tmem_ptr = (uint32_t*)(bars + 5 + 2 * FWD_NS);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nq = (p.S + TR - 1) / TR;
  // blocks of all heads before the next block of any: the longest rows of the whole grid go first
  const int qi = CAUSAL ? nq - 1 - (int)blockIdx.z : (int)blockIdx.z;
  const int h = blockIdx.x, b = blockIdx.y;
  const int n = CAUSAL ? qi + 1 : nq;  // key blocks

  if (tid == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < FWD_NS; ++s) { mbar_init(kv_full + 8 * s, 1); mbar_init(kv_empty + 8 * s, 1); }
    mbar_init(s_full, 1);
    mbar_init(s_free, 8);
    mbar_init(p_ready, 8);
    mbar_init(o_done, 1);
    mbar_fence_init();
  }
  if (warp == 8 && lane == 0) { tma_prefetch_desc(&tq); tma_prefetch_desc(&tk); tma_prefetch_desc(&tv); }
  if (warp == 9) { tmem_alloc(smem_u32(tmem_ptr), 256); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tS = *tmem_ptr, tO = tS + 128;
  pdl_enter();

  if (warp < 8) {
    const int half = warp >> 2, row = (warp & 3) * 32 + lane, q = qi * TR + row;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tSh = tS + lane_off + (uint32_t)(half * 64);  // this thread's 64 scores of a tile
    const uint32_t prow = sP + (uint32_t)half * SLAB_BYTES + (uint32_t)row * 128u;
    float* meet = (float*)(base + TILE_BYTES * (1 + FWD_NS));  // the halves of a row meet in the probability buffer
    // columns of the last tile up to this one count: those above the diagonal of a causal tile, or beyond S, do not
    const int last = (CAUSAL ? row : p.S - 1 - (n - 1) * TR) - half * 64;
    const uint64_t scale2 = pair(p.scale, p.scale);
    bool ok = true;
    float mx = -INFINITY, inv = 0.f;
    int t = 0;  // score tiles over the three passes
    for (; t < n; ++t) {  // pass 1: maximum (rounding is monotonic: the largest is rounded once)
      ok = wait_all(s_full, (uint32_t)t & 1u, p.status, W_ATT_COMPUTE);
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t s[2][32];
      tmem_ld_32x32b_x32(tSh, s[0]);
      tmem_ld_32x32b_x32(tSh + 32, s[1]);
      tmem_ld_wait();
      tc_fence_before_sync();
      warp_arrive(s_free, lane);
      if (t == n - 1) {
        hide(s[0], last);
        hide(s[1], last - 32);
      }
      float m4[4] = {mx, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 64; ++c) m4[c & 3] = fmaxf(m4[c & 3], __uint_as_float(s[c >> 5][c & 31]));
      mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
    }
    meet[half * TR + row] = mx;
    named_bar_sync(1, 256);
    mx = __bfloat162float(__float2bfloat16_rn(fmaxf(mx, meet[(half ^ 1) * TR + row]) * p.scale));
    const uint64_t neg_max = pair(-mx, -mx);
    // pass 2: sum. A warp that walks a row 256 columns at a time, 8 a lane, keeps 32 partial sums: tile j holds those of
    // lanes 16 (j & 1) ... + 15, this thread's columns eight of them. `even` belongs to the current tile, `odd` to the next.
    float even[8], odd[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) even[i] = odd[i] = 0.f;
    for (int j = 0; j < n && ok; ++j, ++t) {
      ok = wait_all(s_full, (uint32_t)t & 1u, p.status, W_ATT_COMPUTE);
      if (!ok) break;
      tc_fence_after_sync();
      const bool edge = j == n - 1;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t s[32];
        tmem_ld_32x32b_x32(tSh + (uint32_t)(hf * 32), s);
        tmem_ld_wait();
        if (hf == 1) {
          tc_fence_before_sync();
          warp_arrive(s_free, lane);
        }
        if (edge) hide(s, last - hf * 32);
#pragma unroll
        for (int e = 0; e < 8; e += 2) {  // the chains of eight sums advance side by side
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int c = i * 8 + e;
            float e0, e1;
            split(exp2x(s[c], s[c + 1], scale2, neg_max), e0, e1);
            even[hf * 4 + i] += e0;
            even[hf * 4 + i] += e1;
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) { const float x = even[i]; even[i] = odd[i]; odd[i] = x; }
    }
    {
      // a warp's butterfly: lanes 16 apart are the two parities, lanes 8 apart the two halves (addition commutes, so both
      // halves get the same sum)
#pragma unroll
      for (int i = 0; i < 8; ++i) meet[(2 + half * 8 + i) * TR + row] = even[i] += odd[i];
      named_bar_sync(1, 256);
#pragma unroll
      for (int i = 0; i < 8; ++i) even[i] += meet[(2 + (half ^ 1) * 8 + i) * TR + row];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; ++i) even[i] += even[i + o];
      inv = 1.f / even[0];
    }
    if (p.row_max && half == 0) {
      const size_t r = ((size_t)b * p.H + h) * p.s_pad + q;
      p.row_max[r] = -mx;
      p.row_inv[r] = inv;
    }
    named_bar_sync(1, 256);  // both have read the other's sums before the buffer takes probabilities
    const uint64_t inv2 = pair(inv, inv);
    for (int j = 0; j < n && ok; ++j, ++t) {  // pass 3: probabilities
      ok = wait_all(s_full, (uint32_t)t & 1u, p.status, W_ATT_COMPUTE);
      if (!ok) break;
      tc_fence_after_sync();
      const bool edge = j == n - 1;
      uint32_t w[32];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t s[32];
        tmem_ld_32x32b_x32(tSh + (uint32_t)(hf * 32), s);
        tmem_ld_wait();
        if (hf == 1) {
          tc_fence_before_sync();
          warp_arrive(s_free, lane);
        }
        if (edge) hide(s, last - hf * 32);
#pragma unroll
        for (int c = 0; c < 32; c += 2) w[hf * 16 + c / 2] = round2(mul2(exp2x(s[c], s[c + 1], scale2, neg_max), inv2));
      }
      if (j > 0) {  // the previous block's P V product has read the probabilities
        ok = wait_all(o_done, (uint32_t)(j - 1) & 1u, p.status, W_ATT_COMPUTE);
        if (!ok) break;
      }
#pragma unroll
      for (int c = 0; c < 8; ++c)
        st_shared_v4(prow + (uint32_t)((c ^ (row & 7)) << 4), w[c * 4], w[c * 4 + 1], w[c * 4 + 2], w[c * 4 + 3]);
      fence_proxy_async_smem();
      warp_arrive(p_ready, lane);
    }
    if (ok) ok = wait_all(o_done, (uint32_t)(n - 1) & 1u, p.status, W_ATT_COMPUTE);
    if (ok) {
      tc_fence_after_sync();
      bf16* out = p.O + (long long)h * p.o_s1 + (long long)b * p.o_s2 + (long long)q * p.ldo + half * 32;
      store_half_row(tO + lane_off + (uint32_t)(half * 32), 1.f, out, q < p.S);
    }
  } else if (warp == 8) {
    if (lane == 0) {
      mbar_arrive_expect_tx(q_full, TILE_BYTES);
      tma_load_4d(sQ, &tq, q_full, 0, qi * TR, h, b);
      for (int i = 0; i < 4 * n; ++i) {
        // i-th tile of the order K0 ... K(n-1), K0 ... K(n-1), K0 K1 V0 K2 V1 ... K(n-1) V(n-2) V(n-1)
        const int i3 = i - 2 * n;
        const bool is_k = i3 <= 0 || ((i3 & 1) && i3 < 2 * n - 1);
        const int j = i3 < 0 ? i % n : is_k ? (i3 + 1) >> 1 : (i3 == 2 * n - 1 ? n - 1 : (i3 >> 1) - 1);
        const int s = i % FWD_NS;
        if (!mbar_wait(kv_empty + 8 * s, ((uint32_t)(i / FWD_NS) & 1u) ^ 1u, p.status, W_ATT_LOAD)) break;
        mbar_arrive_expect_tx(kv_full + 8 * s, TILE_BYTES);
        tma_load_4d(sKV + s * TILE_BYTES, is_k ? &tk : &tv, kv_full + 8 * s, 0, j * TR, h / p.kv_div, b);
      }
    }
  } else {
    if (lane == 0) {
      int i = 0;  // next tile of the ring
      bool ok = mbar_wait(q_full, 0u, p.status, W_ATT_MMA);
      auto next = [&]() {
        ok = ok && mbar_wait(kv_full + 8 * (i % FWD_NS), (uint32_t)(i / FWD_NS) & 1u, p.status, W_ATT_MMA);
        tc_fence_after_sync();
        return sKV + (uint32_t)(i % FWD_NS) * TILE_BYTES;
      };
      for (int t = 0; t < 3 * n + 1 && ok; ++t) {
        if (t < 3 * n) {  // scores: three rounds over the key blocks
          if (t > 0) ok = mbar_wait(s_free, (uint32_t)(t - 1) & 1u, p.status, W_ATT_MMA);
          const uint32_t k = next();
          if (!ok) break;
          mma_scores(tS, sQ, k);
          umma_commit(kv_empty + 8 * (i % FWD_NS));
          umma_commit(s_full);
          ++i;
        }
        if (t > 2 * n) {  // output product of block j
          const int j = t - 2 * n - 1;
          ok = mbar_wait(p_ready, (uint32_t)j & 1u, p.status, W_ATT_MMA);
          const uint32_t v = next();
          if (!ok) break;
          mma_accumulate(tO, sP, v, j == 0);
          umma_commit(kv_empty + 8 * (i % FWD_NS));
          umma_commit(o_done);
          ++i;
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tS, 256);
  }
}

// ---- backward (causal) ----------------------------------------------------------------------------------
// One CTA keeps a pair of resident tiles (R0, R1) and streams pairs (T0, T1):
//   KV = true    R = (K, V) of 128 keys, T = (Q, dO) of the query blocks from the diagonal on; thread row = key
//   KV = false   R = (Q, dO) of 128 queries, T = (K, V) of the key blocks up to the diagonal; thread row = query
// Per streamed block:  s = R0 T0^T,  dp = R1 T1^T,  p = exp(s * scale - max) * inv,  ds = p (dp - dot),
//   acc0 += ds T0  (dK or dQ),   KV: acc1 += p T1  (dV)
// with p and ds of shape [own row][streamed position], K-major operands as the threads write them. The dQ kernel walks
// its blocks twice: the first round only adds up dot = sum p dp, which it leaves for the dK/dV kernel.
// Sixteen compute warps (four per tensor-memory lane quarter, 32 columns each), one TMA warp, one MMA warp; tensor memory:
// s 0-127, dp 128-255, acc0 256-319, acc1 320-383. The next block's s and dp products run while the current block's
// exponentials are taken.
constexpr int BWD_THREADS = 576;
constexpr int BWD_NS = 3;
constexpr int BWD_STAGE_BYTES = 2 * TILE_BYTES + 2048;  // T0, T1, and for KV 128 row maxima, inverse sums and dots
constexpr size_t bwd_smem_bytes(bool kv) {
  return 1024 + (size_t)2 * TILE_BYTES + (size_t)BWD_NS * BWD_STAGE_BYTES + (size_t)(kv ? 4 : 2) * SLAB_BYTES + 128;
}

struct AttBwdParams {
  bf16 *out0, *out1;
  const float *row_max, *row_inv;  // [B*H][s_pad], as row_dot; maxima and dots are stored negated
  float* row_dot;
  int S, s_pad, H, kv_div;
  long long ld, o_s1, o_s2;
  float scale;
  int* status;
};

template <bool KV>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attention_bwd_kernel(const AttBwdParams p, const __grid_constant__ CUtensorMap tr0, const __grid_constant__ CUtensorMap tr1,
                     const __grid_constant__ CUtensorMap tt0, const __grid_constant__ CUtensorMap tt1) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sR = smem_u32(base), sT = sR + 2 * TILE_BYTES, sDS = sT + BWD_NS * BWD_STAGE_BYTES, sP = sDS + 2 * SLAB_BYTES;
  uint64_t* bars = (uint64_t*)(base + 2 * TILE_BYTES + BWD_NS * BWD_STAGE_BYTES + (KV ? 4 : 2) * SLAB_BYTES);
  const uint32_t r_full = smem_u32(bars), t_full = r_full + 8, t_empty = t_full + 8 * BWD_NS, s_full = t_empty + 8 * BWD_NS,
                 s_free = s_full + 8, p_ready = s_free + 8, acc_done = p_ready + 8;
  uint32_t* tmem_ptr = (uint32_t*)(bars + 5 + 2 * BWD_NS);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = (p.S + TR - 1) / TR;
  const int own = KV ? (int)blockIdx.z : nb - 1 - (int)blockIdx.z;  // longest loops of the whole grid first
  const int h = blockIdx.x, b = blockIdx.y, hk = h / p.kv_div;
  const int n = KV ? nb - own : own + 1;
  constexpr int rounds = KV ? 1 : 2;
  const int first = KV ? own : 0;
  const size_t vec_row = ((size_t)b * p.H + h) * p.s_pad;

  if (tid == 0) {
    mbar_init(r_full, 1);
    for (int s = 0; s < BWD_NS; ++s) { mbar_init(t_full + 8 * s, 1); mbar_init(t_empty + 8 * s, 1); }
    mbar_init(s_full, 1);
    mbar_init(s_free, 16);
    mbar_init(p_ready, 16);
    mbar_init(acc_done, 1);
    mbar_fence_init();
  }
  if (warp == 16 && lane == 0) { tma_prefetch_desc(&tr0); tma_prefetch_desc(&tr1); tma_prefetch_desc(&tt0); tma_prefetch_desc(&tt1); }
  if (warp == 17) { tmem_alloc(smem_u32(tmem_ptr), 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tS = *tmem_ptr, tD = tS + 128, tA0 = tS + 256, tA1 = tS + 320;
  pdl_enter();

  if (warp < 16) {
    const int grp = warp >> 2, row = (warp & 3) * 32 + lane;  // columns 32 grp ... + 31 of every tile
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16, col_off = lane_off + (uint32_t)(grp * 32);
    const uint32_t slab = (uint32_t)(grp >> 1) * SLAB_BYTES + (uint32_t)row * 128u;
    const size_t own_row = vec_row + own * TR + row;
    const uint64_t scale2 = pair(p.scale, p.scale);
    uint64_t neg_max = 0, inv2 = 0, neg_dot = 0;
    if (!KV) {
      const float m = p.row_max[own_row], v = p.row_inv[own_row];
      neg_max = pair(m, m);
      inv2 = pair(v, v);
    }
    bool ok = true;
    int t = 0;  // score tiles so far
    if (!KV) {
      // 32 partial sums per row as a warp would keep them (see the forward kernel): this thread has those of its 32
      // columns, four of the current tile's parity and four of the next's
      float even[4], odd[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) even[i] = odd[i] = 0.f;
      for (; t < n; ++t) {
        ok = wait_all(s_full, (uint32_t)t & 1u, p.status, W_ATT_COMPUTE);
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t s[32], dp[32];
        tmem_ld_32x32b_x32(tS + col_off, s);
        tmem_ld_32x32b_x32(tD + col_off, dp);
        tmem_ld_wait();
        tc_fence_before_sync();
        warp_arrive(s_free, lane);
        if (t == n - 1) hide(s, row - grp * 32);  // the block on the diagonal
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int c = i * 8 + e;
            const uint32_t w = round2(mul2(exp2x(s[c], s[c + 1], scale2, neg_max), inv2));
            const uint32_t d = round2(pair(dp[c], dp[c + 1]));
            even[i] = fmaf(__uint_as_float(w << 16), __uint_as_float(d << 16), even[i]);
            even[i] = fmaf(__uint_as_float(w & 0xffff0000u), __uint_as_float(d & 0xffff0000u), even[i]);
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) { const float x = even[i]; even[i] = odd[i]; odd[i] = x; }
      }
      // butterfly: lanes 16 apart are the two parities, 8 and 4 apart the column groups (0 and 2, 1 and 3; then those two
      // sums). The groups meet in the dS operand buffer, which no product reads yet.
      float* meet = (float*)(base + 2 * TILE_BYTES + BWD_NS * BWD_STAGE_BYTES);
#pragma unroll
      for (int i = 0; i < 4; ++i) meet[(grp * 4 + i) * TR + row] = even[i] + odd[i];
      named_bar_sync(1, 512);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        even[i] = (meet[i * TR + row] + meet[(8 + i) * TR + row]) + (meet[(4 + i) * TR + row] + meet[(12 + i) * TR + row]);
      const float dot = -((even[0] + even[2]) + (even[1] + even[3]));
      if (grp == 0) p.row_dot[own_row] = dot;
      neg_dot = pair(dot, dot);
      named_bar_sync(1, 512);  // everyone has read the sums before the buffer takes its first operand
    }
    for (int it = 0; it < n && ok; ++it, ++t) {
      const int st = it % BWD_NS;
      const float* vec = (const float*)(base + 2 * TILE_BYTES + st * BWD_STAGE_BYTES + 2 * TILE_BYTES) + grp * 32;
      if (KV) {  // the row values of the streamed queries came with the tiles
        ok = wait_all(t_full + 8 * st, (uint32_t)(it / BWD_NS) & 1u, p.status, W_ATT_COMPUTE);
        if (!ok) break;
      }
      ok = wait_all(s_full, (uint32_t)t & 1u, p.status, W_ATT_COMPUTE);
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t s[32], dp[32];
      tmem_ld_32x32b_x32(tS + col_off, s);
      tmem_ld_32x32b_x32(tD + col_off, dp);
      tmem_ld_wait();
      tc_fence_before_sync();
      warp_arrive(s_free, lane);
      if (KV ? it == 0 : it == n - 1) {  // the block on the diagonal: a query sees the keys up to its own position
        if (KV) hide_before(s, row - grp * 32);
        else hide(s, row - grp * 32);
      }
      uint32_t wp[16], wd[16];
#pragma unroll
      for (int c = 0; c < 32; c += 2) {
        if (KV) {
          neg_max = *reinterpret_cast<const uint64_t*>(vec + c);
          inv2 = *reinterpret_cast<const uint64_t*>(vec + 128 + c);
          neg_dot = *reinterpret_cast<const uint64_t*>(vec + 256 + c);
        }
        const uint32_t w = round2(mul2(exp2x(s[c], s[c + 1], scale2, neg_max), inv2));
        wp[c >> 1] = w;
        wd[c >> 1] = round2(mul2(widen2(w), add2(widen2(round2(pair(dp[c], dp[c + 1]))), neg_dot)));
      }
      if (it > 0) {  // the previous block's products have read the operands
        ok = wait_all(acc_done, (uint32_t)(it - 1) & 1u, p.status, W_ATT_COMPUTE);
        if (!ok) break;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t off = slab + (uint32_t)((((grp & 1) * 4 + c) ^ (row & 7)) << 4);
        st_shared_v4(sDS + off, wd[c * 4], wd[c * 4 + 1], wd[c * 4 + 2], wd[c * 4 + 3]);
        if (KV) st_shared_v4(sP + off, wp[c * 4], wp[c * 4 + 1], wp[c * 4 + 2], wp[c * 4 + 3]);
      }
      fence_proxy_async_smem();
      warp_arrive(p_ready, lane);
    }
    if (ok) ok = wait_all(acc_done, (uint32_t)(n - 1) & 1u, p.status, W_ATT_COMPUTE);
    if (ok) {
      tc_fence_after_sync();
      const int pos = own * TR + row;
      const uint32_t c0 = (uint32_t)((grp & 1) * 32);
      const long long off = (long long)h * p.o_s1 + (long long)b * p.o_s2 + (long long)pos * p.ld + c0;
      // groups 0 and 1 store the halves of dQ or dK, 2 and 3 those of dV
      if (grp < 2) store_half_row(tA0 + lane_off + c0, p.scale, p.out0 + off, pos < p.S);
      else if (KV) store_half_row(tA1 + lane_off + c0, 1.f, p.out1 + off, pos < p.S);
    }
  } else if (warp == 16) {
    if (lane == 0) {
      mbar_arrive_expect_tx(r_full, 2 * TILE_BYTES);
      tma_load_4d(sR, &tr0, r_full, 0, own * TR, KV ? hk : h, b);
      tma_load_4d(sR + TILE_BYTES, &tr1, r_full, 0, own * TR, KV ? hk : h, b);
      for (int it = 0; it < rounds * n; ++it) {
        const int st = it % BWD_NS, blk = first + it % n;
        const uint32_t bar = t_full + 8 * st, dst = sT + st * BWD_STAGE_BYTES;
        if (!mbar_wait(t_empty + 8 * st, ((uint32_t)(it / BWD_NS) & 1u) ^ 1u, p.status, W_ATT_LOAD)) break;
        mbar_arrive_expect_tx(bar, 2 * TILE_BYTES + (KV ? 1536 : 0));
        tma_load_4d(dst, &tt0, bar, 0, blk * TR, KV ? h : hk, b);
        tma_load_4d(dst + TILE_BYTES, &tt1, bar, 0, blk * TR, KV ? h : hk, b);
        if (KV) {
          bulk_load(dst + 2 * TILE_BYTES, p.row_max + vec_row + blk * TR, 512, bar);
          bulk_load(dst + 2 * TILE_BYTES + 512, p.row_inv + vec_row + blk * TR, 512, bar);
          bulk_load(dst + 2 * TILE_BYTES + 1024, p.row_dot + vec_row + blk * TR, 512, bar);
        }
      }
    }
  } else {
    if (lane == 0) {
      bool ok = mbar_wait(r_full, 0u, p.status, W_ATT_MMA);
      auto scores = [&](int it) {
        ok = ok && mbar_wait(t_full + 8 * (it % BWD_NS), (uint32_t)(it / BWD_NS) & 1u, p.status, W_ATT_MMA);
        if (!ok) return;
        tc_fence_after_sync();
        const uint32_t t = sT + (uint32_t)(it % BWD_NS) * BWD_STAGE_BYTES;
        mma_scores(tS, sR, t);
        mma_scores(tD, sR + TILE_BYTES, t + TILE_BYTES);
        umma_commit(s_full);
      };
      scores(0);
      for (int t = 0; t < rounds * n && ok; ++t) {
        const uint32_t stage = (uint32_t)(t % BWD_NS);
        if (!KV && t < n) umma_commit(t_empty + 8 * stage);  // first round: the tiles are done with when the scores are
        if (t + 1 < rounds * n) {
          ok = mbar_wait(s_free, (uint32_t)t & 1u, p.status, W_ATT_MMA);
          scores(t + 1);
          if (!ok) break;
        }
        if (!KV && t < n) continue;
        const int it = KV ? t : t - n;
        ok = mbar_wait(p_ready, (uint32_t)it & 1u, p.status, W_ATT_MMA);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t tile = sT + stage * BWD_STAGE_BYTES;
        mma_accumulate(tA0, sDS, tile, it == 0);
        if (KV) mma_accumulate(tA1, sP, tile + TILE_BYTES, it == 0);
        umma_commit(t_empty + 8 * stage);
        umma_commit(acc_done);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 17) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tS, 512);
  }
}

int check(const AttentionShape& a) {
  SRT_REQUIRE(a.D == HD && a.S > 0 && a.S % 8 == 0 && a.H > 0 && a.Hkv > 0 && a.H % a.Hkv == 0 && a.B > 0 && a.B <= 65535 && a.S <= 65535 * TR,
              "attention: 64-channel heads, a length that is a multiple of 8 and whole head groups are required");
  return SRT_OK;
}
int tmap(CUtensorMap* tm, const void* p, const AttentionShape& a, int heads, long long ld) {
  return tmap_batched_bf16(tm, p, HD, (uint64_t)a.S, (uint64_t)heads, (uint64_t)a.B, (uint64_t)ld, HD, (uint64_t)(a.S * ld), TR);
}
template <class K>
int reserve_smem(K kernel, size_t bytes) {  // idempotent, cheap: no state of our own to keep per device
  SRT_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return SRT_OK;
}
bool early() { return pdl_big_kernels() && (pdl_classes() & PDL_GEMM) != 0; }

}  // namespace

int attention_s_pad(int S) { return (S + TR - 1) / TR * TR; }

int attention_fwd(const AttentionShape& a, const void* Q, const void* K, const void* V, long long ld_qkv, void* O, long long ld_o,
                  float* rows, float scale, int causal, cudaStream_t st) {
  int rc = check(a);
  if (!rc && !(scale > 0.f)) { set_error("attention: the score scale must be positive"); rc = SRT_ERR_INVALID; }
  if (rc) return rc;
  CUtensorMap tq, tk, tv;
  if ((rc = tmap(&tq, Q, a, a.H, ld_qkv)) || (rc = tmap(&tk, K, a, a.Hkv, ld_qkv)) || (rc = tmap(&tv, V, a, a.Hkv, ld_qkv)))
    return rc;
  SRT_REQUIRE(((uintptr_t)O & 15) == 0 && ld_o % 8 == 0, "attention: unaligned output");
  const int s_pad = attention_s_pad(a.S);
  AttFwdParams p = {(bf16*)O, rows, rows ? rows + (size_t)a.B * a.H * s_pad : nullptr, a.S, s_pad, a.H, a.H / a.Hkv, ld_o, HD,
                    (long long)a.S * ld_o, scale, tc_status_device_ptr()};
  SRT_REQUIRE(p.status != nullptr, "tcgen05 status word unavailable");
  const dim3 grid(a.H, a.B, ceil_div(a.S, TR));
  const size_t smem = fwd_smem_bytes();
  if (causal) {
    if ((rc = reserve_smem(attention_fwd_kernel<true>, smem))) return rc;
    launch_pdl_if(early(), attention_fwd_kernel<true>, grid, dim3(FWD_THREADS), smem, st, p, tq, tk, tv);
  } else {
    if ((rc = reserve_smem(attention_fwd_kernel<false>, smem))) return rc;
    launch_pdl_if(early(), attention_fwd_kernel<false>, grid, dim3(FWD_THREADS), smem, st, p, tq, tk, tv);
  }
  SRT_LAUNCH_CHECK();
  return SRT_OK;
}

int attention_bwd_causal(const AttentionShape& a, const void* Q, const void* K, const void* V, long long ld_qkv, const void* dO,
                         long long ld_o, float* rows, void* dQ, long long ld_dq, void* dK, void* dV, long long ld_dkv,
                         long long dkv_s1, long long dkv_s2, float scale, cudaStream_t st) {
  int rc = check(a);
  if (!rc && !(scale > 0.f)) { set_error("attention: the score scale must be positive"); rc = SRT_ERR_INVALID; }
  if (rc) return rc;
  CUtensorMap tq, tk, tv, tdo;
  if ((rc = tmap(&tq, Q, a, a.H, ld_qkv)) || (rc = tmap(&tk, K, a, a.Hkv, ld_qkv)) || (rc = tmap(&tv, V, a, a.Hkv, ld_qkv)) ||
      (rc = tmap(&tdo, dO, a, a.H, ld_o)))
    return rc;
  SRT_REQUIRE((((uintptr_t)dQ | (uintptr_t)dK | (uintptr_t)dV | (uintptr_t)rows) & 15) == 0 && ld_dq % 8 == 0 && ld_dkv % 8 == 0 &&
                  dkv_s1 % 8 == 0 && dkv_s2 % 8 == 0,
              "attention backward: unaligned tensor");
  const int s_pad = attention_s_pad(a.S);
  const size_t vec = (size_t)a.B * a.H * s_pad;
  AttBwdParams p = {(bf16*)dQ, nullptr, rows, rows + vec, rows + 2 * vec, a.S, s_pad, a.H, a.H / a.Hkv,
                    ld_dq, HD, (long long)a.S * ld_dq, scale, tc_status_device_ptr()};
  SRT_REQUIRE(p.status != nullptr, "tcgen05 status word unavailable");
  const dim3 grid(a.H, a.B, ceil_div(a.S, TR));
  if ((rc = reserve_smem(attention_bwd_kernel<false>, bwd_smem_bytes(false)))) return rc;
  launch_pdl_if(early(), attention_bwd_kernel<false>, grid, dim3(BWD_THREADS), bwd_smem_bytes(false), st, p, tq, tdo, tk, tv);
  SRT_LAUNCH_CHECK();
  p.out0 = (bf16*)dK;
  p.out1 = (bf16*)dV;
  p.ld = ld_dkv;
  p.o_s1 = dkv_s1;
  p.o_s2 = dkv_s2;
  if ((rc = reserve_smem(attention_bwd_kernel<true>, bwd_smem_bytes(true)))) return rc;
  launch_pdl_if(early(), attention_bwd_kernel<true>, grid, dim3(BWD_THREADS), bwd_smem_bytes(true), st, p, tk, tv, tq, tdo);
  SRT_LAUNCH_CHECK();
  return SRT_OK;
}

}  // namespace srt
