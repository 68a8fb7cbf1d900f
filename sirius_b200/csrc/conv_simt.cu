// CUDA-core implicit-GEMM convolution: fp32 accumulate, fp32 or bf16 operands.
//
// This is the exact-arithmetic path (fp32 mode of the training step) and the on-device
// cross-check for the tcgen05 kernels. One gather-GEMM kernel serves fprop and dgrad, one
// split-reduction kernel serves wgrad; partial sums are reduced in a fixed order so results are
// run-to-run deterministic.
#include "common.cuh"
#include "conv_geom.cuh"
#include "ptx.cuh"

namespace srt {

namespace {

constexpr int BM = 64, BN = 64, BK = 16, NT = 256;

template <typename T> struct Ld4;
template <> struct Ld4<float> {
  __device__ static inline void ld(const float* p, float (&v)[4]) {
    float4 r = *reinterpret_cast<const float4*>(p);
    v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
  }
};
template <> struct Ld4<__nv_bfloat16> {
  __device__ static inline void ld(const __nv_bfloat16* p, float (&v)[4]) {
    uint2 r = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(r.x << 16); v[1] = __uint_as_float(r.x & 0xffff0000u);
    v[2] = __uint_as_float(r.y << 16); v[3] = __uint_as_float(r.y & 0xffff0000u);
  }
};

// D[m][n] = sum_k A(m,k) * B[n][k], A gathered from an NHWC tensor (see GatherGeom).
template <typename T>
__global__ void __launch_bounds__(NT)
gather_gemm_simt(GatherGeom g, const T* __restrict__ src, const T* __restrict__ Bm,
                 T* __restrict__ D, const float* __restrict__ bias, const T* addend, const uint8_t* __restrict__ addend_bits) {
  __shared__ __align__(16) float As[BK][BM + 4];
  __shared__ __align__(16) float Bs[BK][BN + 4];
  const int t = threadIdx.x;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int lrow = t >> 2, lk = (t & 3) * 4;

  // fixed per-thread row decode
  const int m = m0 + lrow;
  RowCoord rc = decode_row(g, m);
  const int nb = n0 + lrow;
  const bool nb_ok = nb < g.Nout;
  const T* brow = Bm + (size_t)(nb_ok ? nb : 0) * g.Kg;

  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  const int tx = t & 15, ty = t >> 4;
  for (int k0 = 0; k0 < g.Kg; k0 += BK) {
    const int kk = k0 + lk;
    float a[4] = {0.f, 0.f, 0.f, 0.f}, b[4] = {0.f, 0.f, 0.f, 0.f};
    if (kk < g.Kg) {
      const int tap = kk / g.src_c, c = kk - tap * g.src_c;
      const long long off = m < g.M ? gather_offset(g, rc, tap, c) : -1;
      if (off >= 0) Ld4<T>::ld(src + off, a);
      if (nb_ok) Ld4<T>::ld(brow + kk, b);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) { As[lk + i][lrow] = a[i]; Bs[lk + i][lrow] = b[i]; }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float4 av = *reinterpret_cast<const float4*>(&As[k][ty * 4]);
      float4 bv = *reinterpret_cast<const float4*>(&Bs[k][tx * 4]);
      const float ar[4] = {av.x, av.y, av.z, av.w}, br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(ar[i], br[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int mm = m0 + ty * 4 + i;
    if (mm >= g.M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int nn = n0 + tx * 4 + j;
      if (nn >= g.Nout) continue;
      float v = acc[i][j];
      if (bias) v += bias[nn];
      const size_t o = (size_t)mm * g.Nout + nn;
      if (addend && (!addend_bits || ((addend_bits[o >> 3] >> (o & 7)) & 1))) v += ElemTraits<T>::to_f(addend[o]);
      D[o] = ElemTraits<T>::from_f(v);
    }
  }
}

// partial[split][ko][j] = sum over this split's pixels of dy[pix][ko] * x(pix, j), j = (r,s,c).
template <typename T>
__global__ void __launch_bounds__(NT)
wgrad_simt(GatherGeom g /* fprop geometry: rows = output pixels */, const T* __restrict__ dy,
           const T* __restrict__ x, float* __restrict__ partial, int pix_per_split) {
  __shared__ __align__(16) float As[BK][BM + 4];  // [pix][ko]
  __shared__ __align__(16) float Bs[BK][BN + 4];  // [pix][j]
  const int t = threadIdx.x;
  const int j0 = blockIdx.x * BN, ko0 = blockIdx.y * BM;
  const int Kout = g.Nout, J = g.Kg;
  const int pbeg = blockIdx.z * pix_per_split;
  const int pend = min(g.M, pbeg + pix_per_split);
  const int lp = t >> 4, l4 = (t & 15) * 4;

  const int jj = j0 + l4;
  const bool j_ok = jj < J;
  const int tap = j_ok ? jj / g.src_c : 0, c = j_ok ? jj - tap * g.src_c : 0;
  const int kk = ko0 + l4;
  const bool k_ok = kk < Kout;

  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  const int tx = t & 15, ty = t >> 4;

  for (int p0 = pbeg; p0 < pend; p0 += BK) {
    const int pix = p0 + lp;
    float a[4] = {0.f, 0.f, 0.f, 0.f}, b[4] = {0.f, 0.f, 0.f, 0.f};
    if (pix < pend) {
      if (k_ok) Ld4<T>::ld(dy + (size_t)pix * Kout + kk, a);
      if (j_ok) {
        RowCoord rc = decode_row(g, pix);
        const long long off = gather_offset(g, rc, tap, c);
        if (off >= 0) Ld4<T>::ld(x + off, b);
      }
    }
    *reinterpret_cast<float4*>(&As[lp][l4]) = make_float4(a[0], a[1], a[2], a[3]);
    *reinterpret_cast<float4*>(&Bs[lp][l4]) = make_float4(b[0], b[1], b[2], b[3]);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float4 av = *reinterpret_cast<const float4*>(&As[k][ty * 4]);
      float4 bv = *reinterpret_cast<const float4*>(&Bs[k][tx * 4]);
      const float ar[4] = {av.x, av.y, av.z, av.w}, br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(ar[i], br[j], acc[i][j]);
    }
    __syncthreads();
  }
  float* out = partial + (size_t)blockIdx.z * Kout * J;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int ko = ko0 + ty * 4 + i;
    if (ko >= Kout) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int q = j0 + tx * 4 + j;
      if (q < J) out[(size_t)ko * J + q] = acc[i][j];
    }
  }
}

// ---- fp32 convolution, large tiles -------------------------------------------------------------------------
// D = act(A B^T * scale + shift + addend), A gathered as above (no strided data gradient). Bound by the fp32 pipes: a
// 128 x BN tile per CTA with 8 x (BN / 16) outputs a thread needs 2.7 to 4 fused multiply-adds per shared-memory word
// read, two at a time (fma.rn.f32x2), and the next k-block is fetched into registers while the current one is
// multiplied. Few tiles and a long reduction (deep layers of a small batch) split the reduction over a cluster of CTAs:
// each leaves its tile of partial sums in its shared memory and sums a share of the rows over the cluster, in rank order.
// Unsplit, every output adds the same products in the same order as the 64 x 64 kernel above.
// Batch 5 of ResNet-50 (41 GFLOP of convolutions): 5.09 ms with that kernel (8 TFLOP/s), 1.72 ms with this one.
constexpr int LBM = 128, LBK = 16, LNT = 256;
struct LargeEpilogue {
  const float *scale, *shift, *addend;
  const uint8_t* addend_bits;
  int relu;
};
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t twice(float v) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
template <int BN_>
__global__ void __launch_bounds__(LNT, 2)
gather_gemm_f32_large(const GatherGeom g, const float* __restrict__ src, const float* __restrict__ Bm, float* __restrict__ D,
                      const LargeEpilogue ep, int log2_splits) {
  constexpr int TN = BN_ / 16, NB = BN_ / 64;  // outputs per thread along n; B vectors a thread fetches per k-block
  constexpr int AP = LBM + 4, BP = BN_ + 4;
  extern __shared__ __align__(16) float sm[];  // two stages of A [16][AP] and B [16][BP]; then the tile of partial sums
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  // x: row tiles (2^31 - 1 blocks at most; y and z end at 65535), each as a cluster of `splits` blocks; y: column tiles
  const int splits = 1 << log2_splits, rank = (int)blockIdx.x & (splits - 1);
  const int m0 = ((int)blockIdx.x >> log2_splits) * LBM, n0 = (int)blockIdx.y * BN_;
  const int nkb = (g.Kg + LBK - 1) / LBK;  // below 2^27: the products fit
  const int kb0 = nkb * rank >> log2_splits, kb1 = nkb * (rank + 1) >> log2_splits;
  const int lrow = t >> 2, lk = (t & 3) * 4;

  // two rows of A per thread: the source position of filter tap (0, 0)
  int ih0[2], iw0[2], base[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int m = m0 + lrow + 64 * i;
    const RowCoord rc = decode_row(g, m < g.M ? m : 0);
    ih0[i] = m < g.M ? (g.dgrad ? rc.oh + g.pad : rc.oh * g.stride - g.pad) : -(1 << 20);
    iw0[i] = g.dgrad ? rc.ow + g.pad : rc.ow * g.stride - g.pad;
    base[i] = rc.n * g.src_h;
  }
  const int sgn = g.dgrad ? -1 : 1;
  // filter tap and channel of this thread's four elements of the next k-block
  int kk = kb0 * LBK + lk;
  int tap = kk / g.src_c, c = kk - tap * g.src_c;
  int r = tap / g.S, sf = tap - r * g.S;

  float4 av[2], bv[NB];
  auto fetch = [&]() {
    const bool k_ok = kk < g.Kg;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int ih = ih0[i] + sgn * r, iw = iw0[i] + sgn * sf;
      const bool ok = k_ok && (unsigned)ih < (unsigned)g.src_h && (unsigned)iw < (unsigned)g.src_w;
      av[i] = ok ? *reinterpret_cast<const float4*>(src + ((long long)(base[i] + ih) * g.src_w + iw) * g.src_c + c)
                 : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int n = n0 + lrow + 64 * i;
      bv[i] = k_ok && n < g.Nout ? *reinterpret_cast<const float4*>(Bm + (size_t)n * g.Kg + kk) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    kk += LBK;
    c += LBK;
    while (c >= g.src_c) {
      c -= g.src_c;
      if (++sf == g.S) { sf = 0; ++r; }
    }
  };
  auto stash = [&](int st) {
    float* A = sm + st * LBK * (AP + BP);
    float* B = A + LBK * AP;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float v[4] = {av[i].x, av[i].y, av[i].z, av[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) A[(lk + e) * AP + lrow + 64 * i] = v[e];
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const float v[4] = {bv[i].x, bv[i].y, bv[i].z, bv[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) B[(lk + e) * BP + lrow + 64 * i] = v[e];
    }
  };
  uint64_t acc[8][TN / 2];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
  if (kb0 < kb1) { fetch(); stash(0); }
  __syncthreads();
  for (int kb = kb0; kb < kb1; ++kb) {
    const int st = (kb - kb0) & 1;
    const bool more = kb + 1 < kb1;
    if (more) fetch();
    const float* A = sm + st * LBK * (AP + BP);
    const float* B = A + LBK * AP;
#pragma unroll
    for (int k = 0; k < LBK; ++k) {
      const float4 a0 = *reinterpret_cast<const float4*>(A + k * AP + ty * 4), a1 = *reinterpret_cast<const float4*>(A + k * AP + 64 + ty * 4);
      const uint64_t a[8] = {twice(a0.x), twice(a0.y), twice(a0.z), twice(a0.w), twice(a1.x), twice(a1.y), twice(a1.z), twice(a1.w)};
      uint64_t b[TN / 2];
#pragma unroll
      for (int j = 0; j < TN / 4; ++j) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(B + k * BP + j * 64 + tx * 4);
        b[2 * j] = v.x;
        b[2 * j + 1] = v.y;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma2(a[i], b[j], acc[i][j]);
    }
    if (more) stash(st ^ 1);
    __syncthreads();
  }
  auto finish = [&](int mm, int nn, float4 v) {  // four columns; Nout is a multiple of four
    if (mm >= g.M || nn >= g.Nout) return;
    const size_t o = (size_t)mm * g.Nout + nn;
    float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (ep.scale) f[e] *= ep.scale[nn + e];
      if (ep.shift) f[e] += ep.shift[nn + e];
      if (ep.addend && (!ep.addend_bits || ((ep.addend_bits[(o + e) >> 3] >> ((o + e) & 7)) & 1))) f[e] += ep.addend[o + e];
      if (ep.relu) f[e] = fmaxf(f[e], 0.f);
    }
    *reinterpret_cast<float4*>(D + o) = make_float4(f[0], f[1], f[2], f[3]);
  };
  // row i of this thread: ty * 4 + i (i < 4), 64 + ty * 4 + i - 4; column group j: j * 64 + tx * 4
  auto quad = [&](int i, int j) {
    float4 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(acc[i][2 * j]));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.z), "=f"(v.w) : "l"(acc[i][2 * j + 1]));
    return v;
  };
  if (splits == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < TN / 4; ++j)
        finish(m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4), n0 + j * 64 + tx * 4, quad(i, j));
    return;
  }
  // the loop's last barrier has passed: the stages are free for the tile of partial sums [128][BN_]
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < TN / 4; ++j)
      *reinterpret_cast<float4*>(sm + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4) * BN_ + j * 64 + tx * 4) = quad(i, j);
  ptx::cluster_sync_all();
  const int share = LBM >> log2_splits;  // rows this CTA finishes
  for (int q = t; q < share * (BN_ / 4); q += LNT) {
    const int row = rank * share + q / (BN_ / 4), col = (q % (BN_ / 4)) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < splits; ++s) {
      const float4 x = ptx::ld_cluster_f4(ptx::map_to_cta(ptx::smem_u32(sm + row * BN_ + col), (uint32_t)s));
      v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
    }
    finish(m0 + row, n0 + col, v);
  }
  ptx::cluster_sync_all();  // nobody leaves while its sums are still read
}

// Tile width and cluster size. 128 columns where the output has as many and the cluster can still fill the device; a
// reduction is split while the grid stays within two CTAs per SM and every part keeps four k-blocks. Clusters beyond a CTA
// pair only on the whole device: a partition of it may have no room for one.
struct LargePlan { int bn, log2_splits; };
LargePlan plan_large(const GatherGeom& g, bool may_split) {
  const int mt = ceil_div(g.M, LBM), nkb = ceil_div(g.Kg, LBK), room = 2 * sm_count();
  const int most = !may_split ? 0 : sm_limit() == 0 ? 3 : 1;  // log2 of the largest cluster
  LargePlan p;
  p.bn = g.Nout > 64 && ((long long)mt * ceil_div(g.Nout, 128) << most) >= sm_count() ? 128 : 64;
  const long long tiles = (long long)mt * ceil_div(g.Nout, p.bn);
  p.log2_splits = most;
  while (p.log2_splits > 0 && (tiles << p.log2_splits > room || nkb < 4 << p.log2_splits)) --p.log2_splits;
  return p;
}
template <int BN_>
int launch_large(const GatherGeom& g, const float* src, const float* Bm, float* D, const LargeEpilogue& ep, int log2_splits,
                 cudaStream_t st) {
  const int splits = 1 << log2_splits;
  constexpr size_t stages = 2 * LBK * (LBM + 4 + BN_ + 4) * sizeof(float), tile = LBM * BN_ * sizeof(float);
  constexpr size_t smem = stages > tile ? stages : tile;
  SRT_CHECK_CUDA(cudaFuncSetAttribute(gather_gemm_f32_large<BN_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ceil_div(g.M, LBM) * splits, ceil_div(g.Nout, BN_));
  cfg.blockDim = dim3(LNT);
  cfg.dynamicSmemBytes = splits > 1 ? smem : stages;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = splits > 1 ? 1 : 0;
  SRT_CHECK_CUDA(cudaLaunchKernelEx(&cfg, gather_gemm_f32_large<BN_>, g, src, Bm, D, ep, log2_splits));
  SRT_LAUNCH_CHECK();
  return SRT_OK;
}
// The large-tile kernel reads and writes whole 16-byte vectors. Column tiles lie on grid y.
bool large_shape_ok(const GatherGeom& g) {
  return (!g.dgrad || g.stride == 1) && g.src_c % 4 == 0 && g.Kg % 4 == 0 && g.Nout % 4 == 0 && ceil_div(g.Nout, 64) <= 65535;
}
bool large_ok(const GatherGeom& g, const void* src, const void* Bm, const void* D) {
  return large_shape_ok(g) && (((uintptr_t)src | (uintptr_t)Bm | (uintptr_t)D) & 15) == 0;
}
int conv_large(const GatherGeom& g, const void* src, const void* Bm, void* D, const LargeEpilogue& ep, bool may_split,
               cudaStream_t st) {
  const LargePlan p = plan_large(g, may_split);
  return p.bn == 128 ? launch_large<128>(g, (const float*)src, (const float*)Bm, (float*)D, ep, p.log2_splits, st)
                     : launch_large<64>(g, (const float*)src, (const float*)Bm, (float*)D, ep, p.log2_splits, st);
}

}  // namespace

// Partial sums out of L2, added in split order with eight splits in flight. VEC: four elements a thread, where that still
// leaves every SM a block; otherwise (small filters, odd counts) an element a thread.
template <bool VEC>
__global__ void split_reduce_kernel(const float* __restrict__ partial, float* __restrict__ out,
                                    long long n, int splits) {
  pdl_enter();
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  if constexpr (VEC) {
    const float4* p4 = reinterpret_cast<const float4*>(partial);
    const long long n4 = n / 4;
    for (; i < n4; i += stride) {
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
      int k = 0;
      for (; k + 8 <= splits; k += 8) {
        float4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = p4[(k + u) * n4 + i];
#pragma unroll
        for (int u = 0; u < 8; ++u) { s.x += v[u].x; s.y += v[u].y; s.z += v[u].z; s.w += v[u].w; }
      }
#pragma unroll 4
      for (; k < splits; ++k) {
        const float4 v = p4[k * n4 + i];
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
      reinterpret_cast<float4*>(out)[i] = s;
    }
  } else {
    for (; i < n; i += stride) {
      float s = 0.f;
      int k = 0;
      for (; k + 8 <= splits; k += 8) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = partial[(size_t)(k + u) * n + i];
#pragma unroll
        for (int u = 0; u < 8; ++u) s += v[u];
      }
      for (; k < splits; ++k) s += partial[(size_t)k * n + i];
      out[i] = s;
    }
  }
}

int launch_split_reduce(const float* partial, float* out, long long n, int splits,
                        cudaStream_t st) {
  const int threads = 256;
  const bool vec = n % 4 == 0 && (((uintptr_t)partial | (uintptr_t)out) & 15) == 0 && n / 4 >= (long long)threads * sm_count();
  long long blocks = ((vec ? n / 4 : n) + threads - 1) / threads;
  const long long cap = (long long)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  launch_pdl(vec ? split_reduce_kernel<true> : split_reduce_kernel<false>, dim3((unsigned)blocks), dim3(threads), 0, st, partial, out,
             n, splits);
  SRT_LAUNCH_CHECK();
  return SRT_OK;
}

template <typename T>
static int gather_gemm_simt_launch(const GatherGeom& g, const void* src, const void* Bm, void* D,
                                   const srt_conv_epilogue* ep, cudaStream_t st) {
  dim3 grid(ceil_div(g.M, BM), ceil_div(g.Nout, BN));
  gather_gemm_simt<T><<<grid, NT, 0, st>>>(g, (const T*)src, (const T*)Bm, (T*)D,
                                          ep ? ep->bias : nullptr,
                                          ep ? (const T*)ep->addend : nullptr, ep ? ep->addend_bits : nullptr);
  SRT_LAUNCH_CHECK();
  return SRT_OK;
}

int conv_gather_gemm_simt(const GatherGeom& g, int dtype, const void* src, const void* Bm, void* D,
                          const srt_conv_epilogue* ep, cudaStream_t st) {
  SRT_REQUIRE(g.src_c % 4 == 0, "simt conv: channels per tap (%d) must be a multiple of 4", g.src_c);
  if (dtype == SRT_F32 && large_ok(g, src, Bm, D)) {
    const LargeEpilogue e = {nullptr, ep ? ep->bias : nullptr, ep ? (const float*)ep->addend : nullptr,
                             ep && ep->addend ? ep->addend_bits : nullptr, 0};
    return conv_large(g, src, Bm, D, e, false, st);
  }
  if (dtype == SRT_F32) return gather_gemm_simt_launch<float>(g, src, Bm, D, ep, st);
  return gather_gemm_simt_launch<__nv_bfloat16>(g, src, Bm, D, ep, st);
}

bool conv_infer_simt_ok(const GatherGeom& g) { return large_shape_ok(g); }
int conv_infer_simt(const GatherGeom& g, const void* src, const void* Bm, void* D, const InferEpilogue& ep, cudaStream_t st) {
  SRT_REQUIRE(large_ok(g, src, Bm, D), "conv: unaligned tensor");
  const LargeEpilogue e = {ep.scale, ep.shift, (const float*)ep.addend, nullptr, ep.act == ACT_RELU};
  return conv_large(g, src, Bm, D, e, true, st);
}

int wgrad_simt_splits(const GatherGeom& g) {
  const int tiles = ceil_div(g.Nout, BM) * ceil_div(g.Kg, BN);
  int want = ceil_div(4 * sm_count(), tiles);
  int max_by_pix = ceil_div(g.M, 4 * BK);
  int splits = want < max_by_pix ? want : max_by_pix;
  if (splits < 1) splits = 1;
  if (splits > 256) splits = 256;
  return splits;
}

size_t conv_wgrad_simt_scratch_bytes(const GatherGeom& g) {
  const int splits = wgrad_simt_splits(g);
  return splits > 1 ? (size_t)splits * g.Nout * g.Kg * sizeof(float) : 0;
}

int conv_wgrad_simt(const GatherGeom& g, int dtype, const void* dy, const void* x, float* dw,
                    void* scratch, size_t scratch_bytes, cudaStream_t st) {
  SRT_REQUIRE(g.src_c % 4 == 0 && g.Nout % 4 == 0,
              "simt wgrad: C (%d) and K (%d) must be multiples of 4", g.src_c, g.Nout);
  int splits = wgrad_simt_splits(g);
  const size_t need = conv_wgrad_simt_scratch_bytes(g);
  SRT_REQUIRE(scratch_bytes >= need && (need == 0 || scratch != nullptr),
              "simt wgrad: scratch too small (%zu < %zu)", scratch_bytes, need);
  int pps = ceil_div(ceil_div(g.M, splits), BK) * BK;
  splits = ceil_div(g.M, pps);
  float* partial = splits > 1 ? (float*)scratch : dw;
  dim3 grid(ceil_div(g.Kg, BN), ceil_div(g.Nout, BM), splits);
  if (dtype == SRT_F32)
    wgrad_simt<float><<<grid, NT, 0, st>>>(g, (const float*)dy, (const float*)x, partial, pps);
  else
    wgrad_simt<__nv_bfloat16><<<grid, NT, 0, st>>>(g, (const __nv_bfloat16*)dy,
                                                    (const __nv_bfloat16*)x, partial, pps);
  SRT_LAUNCH_CHECK();
  if (splits > 1) return launch_split_reduce(partial, dw, (long long)g.Nout * g.Kg, splits, st);
  return SRT_OK;
}

}  // namespace srt
