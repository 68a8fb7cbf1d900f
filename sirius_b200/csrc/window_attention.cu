// Shifted-window attention (Swin) of one window and head per block, forward and backward, straight from and to the fused
// projection [tokens][3][heads][32]: no windowed copies, no score matrices, no transposes in memory.
//
// A window of at most 64 tokens with 32 channels per head is one 64 x 64 score tile: four warps of 16 rows keep it in
// registers as mma.sync m16n8k16 accumulators (2 x 8 of them per warp and product: 0.3 MFLOP per window and head against
// 9 KB of operands, so the legacy tensor path is far from being the limit and a 128-row tcgen05 tile would be half
// empty). What bounds it is moving Q, K, V, the output and their gradients once: 77 MB in and 26 MB out for 32 images
// of the first stage. The previous path (gather to windows, batched GEMM, softmax, padded transposes, batched GEMMs, scatter)
// moved each of them several times and ran one 128-row tile per window and head.
// Rounding points and orders of sums are those of that path: scores, probabilities, dP and dS are bf16, everything
// between fp32.
#include "common.cuh"
#include "ops.cuh"
#include "window_geom.cuh"

namespace srt {

namespace {

using bf16 = __nv_bfloat16;
constexpr int WT = 128;        // threads: four warps of 16 rows
constexpr int MAXL = 64;       // tokens of a window, padded
constexpr int HD = 32;         // channels of a head
constexpr int TP = HD * 2 + 16;    // row pitch of a [64][32] tile in bytes: ldmatrix reads eight rows from 32 different banks
constexpr int PP = MAXL * 2 + 16;  // ... of a [64][64] tile
constexpr int TILE = MAXL * TP, PTILE = MAXL * PP;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ uint32_t pack(float lo, float hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float lo_f(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// Sum over a row of per-column values that already hold columns j and j + 32: in the order of a warp's butterfly with one
// such column a lane (lanes 16 and 8 apart are tiles of this thread, 4 and 2 apart the other threads of its quad, 1 apart
// the two columns of a tile). Addition commutes, so the four threads get the same sum.
__device__ __forceinline__ float row_sum(const float (&p)[4][2]) {
  float s[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    s[e] = (p[0][e] + p[2][e]) + (p[1][e] + p[3][e]);
    s[e] += __shfl_xor_sync(0xffffffffu, s[e], 2);
    s[e] += __shfl_xor_sync(0xffffffffu, s[e], 1);
  }
  return s[0] + s[1];
}
// c[16 rows of the warp][64] += A rows (tile `a`, [row][32]) times B^T (tile `b`, [64][32])
__device__ __forceinline__ void product_rows(float (&c)[8][4], uint32_t a, uint32_t b, int warp, int lane) {
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    uint32_t af[4];
    ldsm4(a + (uint32_t)(warp * 16 + (lane & 15)) * TP + (uint32_t)(k * 32 + (lane >> 4) * 16), af);
#pragma unroll
    for (int n = 0; n < 4; ++n) {  // pairs of 8-column tiles
      uint32_t bf[4];
      ldsm4(b + (uint32_t)(n * 16 + (lane >> 4) * 8 + (lane & 7)) * TP + (uint32_t)(k * 32 + ((lane >> 3) & 1) * 16), bf);
      mma(c[2 * n], af, bf[0], bf[1]);
      mma(c[2 * n + 1], af, bf[2], bf[3]);
    }
  }
}
// c[16 rows][32] += A (fragments, 64 columns) times B (tile `b`, [64][32])
__device__ __forceinline__ void product_cols(float (&c)[4][4], const uint32_t (&a)[4][4], uint32_t b, int lane) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      uint32_t bf[4];
      ldsm4t(b + (uint32_t)(k * 16 + (lane & 15)) * TP + (uint32_t)(n * 32 + (lane >> 4) * 16), bf);
      mma(c[2 * n], a[k], bf[0], bf[1]);
      mma(c[2 * n + 1], a[k], bf[2], bf[3]);
    }
  }
}
// fragments of the 16 rows `row0` of M^T for a [64][64] tile M
__device__ __forceinline__ void transposed(uint32_t (&a)[4][4], uint32_t m, int row0, int lane) {
#pragma unroll
  for (int k = 0; k < 4; ++k)
    ldsm4t(m + (uint32_t)(k * 16 + (lane >> 4) * 8 + (lane & 7)) * PP + (uint32_t)((row0 + ((lane >> 3) & 1) * 8) * 2), a[k]);
}

struct WinAttParams {
  WinGeom g;
  int heads, L;
  float scale;
  const bf16* qkv;    // [tokens][3][heads][32]
  const float* table; // [(2 WS - 1)^2][heads]
  bf16* out;          // forward: [tokens][heads][32]
  const bf16* dout;   // backward
  bf16 *dqkv, *dS;    // dS: [windows][heads][L][ld]
  int ld;
};

// Shared state of a block: token rows, table column of the head, bias offsets and shift regions of the columns.
struct WinShared {
  int row[MAXL];
  int col[MAXL];      // jy * (2 WS - 1) + jx
  int region[MAXL];
  float bias[15 * 15];
};
__device__ __forceinline__ void win_setup(WinShared& s, const WinAttParams& p, int64_t win, int hd) {
  const int t = threadIdx.x, WS = p.g.WS, side = 2 * WS - 1;
  for (int i = t; i < side * side; i += WT) s.bias[i] = p.table[i * p.heads + hd];
  if (t < MAXL) {
    const int tok = t < p.L ? t : 0, y = tok / WS, x = tok - y * WS;
    s.row[t] = (int)win_token_to_natural(p.g, win, tok);
    s.col[t] = y * side + x;
    const int wx = (int)(win % p.g.nWx), wy = (int)((win / p.g.nWx) % p.g.nWy);
    s.region[t] = p.g.shift > 0 ? shift_region(wy * WS + y, p.g.Hs, WS, p.g.shift) * 3 + shift_region(wx * WS + x, p.g.Ws, WS, p.g.shift) : 0;
  }
}
// One [L][32] tile into shared memory, the rows up to 64 as zeros.
__device__ __forceinline__ void load_tile(uint8_t* tile, const bf16* src, int ld, const WinShared& s, int L) {
  for (int i = threadIdx.x; i < MAXL * 4; i += WT) {
    const int tok = i >> 2, v = i & 3;
    uint8_t* d = tile + tok * TP + v * 16;
    if (tok < L) copy16(smem_addr(d), src + (int64_t)s.row[tok] * ld + v * 8);
    else *reinterpret_cast<uint4*>(d) = make_uint4(0, 0, 0, 0);
  }
}
// Probabilities of this warp's 16 rows as bf16 A fragments: P = softmax(bf16(Q K^T * scale) + bias + mask).
__device__ __forceinline__ void probabilities(uint32_t (&pf)[4][4], const WinShared& s, const WinAttParams& p, uint32_t sq, uint32_t sk,
                                              int warp, int lane) {
  float c[8][4];
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) c[n][e] = 0.f;
  product_rows(c, sq, sk, warp, lane);
  const int side = 2 * p.g.WS - 1, origin = (p.g.WS - 1) * side + p.g.WS - 1;
  const int r0 = warp * 16 + (lane >> 2);
  int rofs[2], rreg[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) { rofs[h] = s.col[r0 + 8 * h] + origin; rreg[h] = s.region[r0 + 8 * h]; }
  float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
  for (int n = 0; n < 8; ++n) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int j = n * 8 + (lane & 3) * 2 + e, cj = s.col[j], gj = s.region[j];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float v = -INFINITY;
        if (j < p.L) {
          v = __bfloat162float(__float2bfloat16_rn(c[n][2 * h + e] * p.scale)) + s.bias[rofs[h] - cj];
          if (gj != rreg[h]) v += -100.f;
        }
        c[n][2 * h + e] = v;
        mx[h] = fmaxf(mx[h], v);
      }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
    mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
  }
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) c[n][e] = __expf(c[n][e] - mx[e >> 1]);
  float sum[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float part[4][2];
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) part[n][e] = c[n][2 * h + e] + c[n + 4][2 * h + e];
    sum[h] = 1.f / row_sum(part);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h) pf[k][t * 2 + h] = pack(c[2 * k + t][2 * h] * sum[h], c[2 * k + t][2 * h + 1] * sum[h]);
}
// Accumulators of 16 rows x 32 channels, scaled, through this warp's rows of a tile in shared memory to the token rows.
__device__ __forceinline__ void store_rows(float (&c)[4][4], float scale, uint8_t* tile, bf16* dst, int ld, const WinShared& s, int L,
                                           int warp, int lane) {
  const int r0 = warp * 16 + (lane >> 2);
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      *reinterpret_cast<uint32_t*>(tile + (r0 + 8 * h) * TP + n * 16 + (lane & 3) * 4) = pack(c[n][2 * h] * scale, c[n][2 * h + 1] * scale);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int tok = warp * 16 + (lane >> 2) + 8 * i, v = lane & 3;
    if (tok < L) *reinterpret_cast<uint4*>(dst + (int64_t)s.row[tok] * ld + v * 8) = *reinterpret_cast<const uint4*>(tile + tok * TP + v * 16);
  }
}

__global__ void __launch_bounds__(WT)
window_attention_fwd_kernel(const WinAttParams p) {
  __shared__ __align__(16) uint8_t tiles[3 * TILE];
  __shared__ WinShared s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hd = blockIdx.x % p.heads, C = p.heads * HD;
  const int64_t win = blockIdx.x / p.heads;
  pdl_enter();
  win_setup(s, p, win, hd);
  __syncthreads();
  for (int i = 0; i < 3; ++i) load_tile(tiles + i * TILE, p.qkv + i * C + hd * HD, 3 * C, s, p.L);
  copies_done();
  __syncthreads();
  const uint32_t sq = smem_addr(tiles), sk = sq + TILE, sv = sk + TILE;
  uint32_t pf[4][4];
  probabilities(pf, s, p, sq, sk, warp, lane);
  float o[4][4] = {};
  product_cols(o, pf, sv, lane);
  store_rows(o, 1.f, tiles, p.out + hd * HD, C, s, p.L, warp, lane);  // Q's tile: a warp reads and writes only its own rows of it
}

__global__ void __launch_bounds__(WT)
window_attention_bwd_kernel(const WinAttParams p) {
  __shared__ __align__(16) uint8_t tiles[4 * TILE];
  __shared__ __align__(16) uint8_t mats[2 * PTILE];  // P and dS, [query][key]
  __shared__ WinShared s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hd = blockIdx.x % p.heads, C = p.heads * HD;
  const int64_t win = blockIdx.x / p.heads;
  pdl_enter();
  win_setup(s, p, win, hd);
  __syncthreads();
  for (int i = 0; i < 3; ++i) load_tile(tiles + i * TILE, p.qkv + i * C + hd * HD, 3 * C, s, p.L);
  load_tile(tiles + 3 * TILE, p.dout + hd * HD, C, s, p.L);
  copies_done();
  __syncthreads();
  const uint32_t sq = smem_addr(tiles), sk = sq + TILE, sv = sk + TILE, sdo = sv + TILE;
  uint32_t pf[4][4], df[4][4];
  probabilities(pf, s, p, sq, sk, warp, lane);
  {
    float c[8][4] = {};
    product_rows(c, sdo, sv, warp, lane);  // dP = dO V^T
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) df[k][t * 2 + h] = pack(c[2 * k + t][2 * h], c[2 * k + t][2 * h + 1]);
    float dot[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float part[4][2];
#pragma unroll
      for (int n = 0; n < 4; ++n) {  // columns of tile n, then those 32 further, in tile n + 4
        const uint32_t w0 = pf[n >> 1][(n & 1) * 2 + h], d0 = df[n >> 1][(n & 1) * 2 + h];
        const uint32_t w1 = pf[2 + (n >> 1)][(n & 1) * 2 + h], d1 = df[2 + (n >> 1)][(n & 1) * 2 + h];
        part[n][0] = fmaf(lo_f(w1), lo_f(d1), fmaf(lo_f(w0), lo_f(d0), 0.f));
        part[n][1] = fmaf(hi_f(w1), hi_f(d1), fmaf(hi_f(w0), hi_f(d0), 0.f));
      }
      dot[h] = row_sum(part);
    }
    const int r0 = warp * 16 + (lane >> 2);
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t d = df[k][t * 2 + h], w = pf[k][t * 2 + h];
          const uint32_t ds = pack(lo_f(w) * (lo_f(d) - dot[h]), hi_f(w) * (hi_f(d) - dot[h]));
          df[k][t * 2 + h] = ds;
          uint8_t* m = mats + (r0 + 8 * h) * PP + ((2 * k + t) * 8 + (lane & 3) * 2) * 2;
          *reinterpret_cast<uint32_t*>(m) = w;
          *reinterpret_cast<uint32_t*>(m + PTILE) = ds;
        }
  }
  float dq[4][4] = {};
  product_cols(dq, df, sk, lane);  // dQ = dS K * scale
  __syncthreads();                 // P and dS are whole; every warp is done with K and V
  const uint32_t sp = smem_addr(mats);
  uint32_t a[4][4];
  float dv[4][4] = {}, dk[4][4] = {};
  transposed(a, sp, warp * 16, lane);
  product_cols(dv, a, sdo, lane);  // dV = P^T dO
  transposed(a, sp + PTILE, warp * 16, lane);
  product_cols(dk, a, sq, lane);   // dK = dS^T Q * scale
  // dS for the gradient of the bias table: whole rows, the pad columns as zeros (their probabilities are)
  bf16* ds = p.dS + (win * p.heads + hd) * (int64_t)p.L * p.ld;
  for (int i = threadIdx.x; i < p.L * (p.ld / 8); i += WT) {
    const int r = i / (p.ld / 8), v = i - r * (p.ld / 8);
    *reinterpret_cast<uint4*>(ds + r * p.ld + v * 8) = *reinterpret_cast<const uint4*>(mats + PTILE + r * PP + v * 16);
  }
  __syncthreads();  // every warp is done with Q and dO
  bf16* dst = p.dqkv + hd * HD;
  store_rows(dq, p.scale, tiles, dst, 3 * C, s, p.L, warp, lane);
  store_rows(dk, p.scale, tiles + TILE, dst + C, 3 * C, s, p.L, warp, lane);
  store_rows(dv, 1.f, tiles + 2 * TILE, dst + 2 * C, 3 * C, s, p.L, warp, lane);
}

int window_params(WinAttParams& p, const WindowShape& w, int heads, int D, const void* qkv, const float* table, float scale) {
  SRT_REQUIRE(w.B > 0 && w.WS > 0 && w.Hs % w.WS == 0 && w.Ws % w.WS == 0 && w.shift >= 0 && w.shift < w.WS && heads > 0,
              "window attention: the map (%d x %d) must be a multiple of the window (%d)", w.Hs, w.Ws, w.WS);
  SRT_REQUIRE(window_attention_supported(w.WS, D) && ((uintptr_t)qkv & 15) == 0,
              "window attention: 32-channel heads and windows of at most 64 tokens");
  SRT_REQUIRE((long long)w.B * w.Hs * w.Ws < (1ll << 31) && (long long)w.B * (w.Hs / w.WS) * (w.Ws / w.WS) * heads < (1ll << 31),
              "window attention: too many tokens or windows");
  p = {};
  p.g = {w.B, w.Hs, w.Ws, w.WS, w.shift, w.Hs / w.WS, w.Ws / w.WS};
  p.heads = heads;
  p.L = w.WS * w.WS;
  p.scale = scale;
  p.qkv = (const bf16*)qkv;
  p.table = table;
  return SRT_OK;
}

}  // namespace

int window_attention_fwd(const void* qkv, const float* table, void* out, const WindowShape& w, int heads, int D, float scale,
                         cudaStream_t st) {
  WinAttParams p;
  if (int rc = window_params(p, w, heads, D, qkv, table, scale)) return rc;
  SRT_REQUIRE(((uintptr_t)out & 15) == 0, "window attention: unaligned output");
  p.out = (bf16*)out;
  launch_pdl(window_attention_fwd_kernel, dim3((unsigned)(w.B * p.g.nWy * p.g.nWx * heads)), dim3(WT), 0, st, p);
  SRT_LAUNCH_CHECK();
  return SRT_OK;
}
int window_attention_bwd(const void* qkv, const float* table, const void* dout, void* dqkv, void* dS, int ld, const WindowShape& w,
                         int heads, int D, float scale, cudaStream_t st) {
  WinAttParams p;
  if (int rc = window_params(p, w, heads, D, qkv, table, scale)) return rc;
  SRT_REQUIRE((((uintptr_t)dout | (uintptr_t)dqkv | (uintptr_t)dS) & 15) == 0 && ld % 8 == 0 && ld >= p.L && ld <= MAXL,
              "window attention: unaligned gradient or bad row pitch %d", ld);
  p.dout = (const bf16*)dout;
  p.dqkv = (bf16*)dqkv;
  p.dS = (bf16*)dS;
  p.ld = ld;
  launch_pdl(window_attention_bwd_kernel, dim3((unsigned)(w.B * p.g.nWy * p.g.nWx * heads)), dim3(WT), 0, st, p);
  SRT_LAUNCH_CHECK();
  return SRT_OK;
}

}  // namespace srt
