// Tall-skinny Gram products C(p x q) = A(N x p)^T B(N x q) of FP32 vectors on
// the 5th-generation tensor cores: the Rayleigh matrix V^T (HV) (calcrmat,
// block_davidson.f90:954-967), the projections of the block
// orthogonalisation (subspace_projection / qrortho, :1226-1284, 1423-1465)
// and their Gram matrices, on the FP32 phases of the mixed-precision ladder.
//
// Precision.  Every FP32 value x is split into three BF16 slices
// x = x0 + x1 + x2 (x0 = bf16(x), x1 = bf16(x - x0), x2 = bf16(x - x0 - x1);
// the differences are exact in FP32), and the six slice products whose
// weight is at least 2^-18 (x0y0, x0y1, x1y0, x0y2, x1y1, x2y0) are
// accumulated by tcgen05.mma (kind::f16, FP32 accumulate in TMEM).  The
// dropped products are below 2^-26 of |x||y|, so each product carries about
// FP32 rounding.  A TMEM accumulator sums 128 rows; the epilogue adds it into
// double-float registers (df.h), and the per-block partials are summed in
// FP64 in a fixed order, as the CUDA-core kernel of dense.cu does.
//
// One CTA per (row block, 128-column tile of A), warp-specialised: 16 producer
// warps hold the next two 64-row stages of their columns in registers, split
// them and store the slices into a 3-stage ring of 128-byte-swizzled K-major
// operand tiles; one warp issues the MMAs (24 per stage, by an elected lane:
// one thread walking them alone took about 200 cycles each, 165 us a product
// of any p <= 128 at N = 610,000); eight warps drain the accumulator every 128
// rows.  TMEM holds two accumulators, so the MMAs of the next 128 rows run
// while one is drained.
// Every wait is bounded; a wait that gives up sets the error word and the
// call returns ADCGPU_DEVICE_TIMEOUT.
#include <cuda_bf16.h>

#include <algorithm>

#include "dense.h"
#include "df.h"
#include "internal.h"
#include "umma.h"

namespace adcgpu {

using namespace umma;

namespace {

constexpr int GU_WARPS = 16;   // producer warps
constexpr int GU_THREADS = 32 * (GU_WARPS + 8 + 1);   // and 8 drain warps, 1 MMA issuer
constexpr int GU_M = 128;      // A columns per CTA (MMA M)
constexpr int GU_K = 64;       // rows per stage: one 128-byte swizzled row of 64 BF16 values
constexpr int GU_NS = 3;       // ring stages
constexpr int GU_F = 2;        // stages summed per TMEM accumulator before it is drained
constexpr int GU_A_SLICE = GU_M * 128;   // bytes of one slice of the A tile

template <int NQ>
__host__ __device__ constexpr int gu_stage_bytes() { return 3 * GU_A_SLICE + 3 * NQ * 128; }

template <int NQ>
__host__ __device__ constexpr uint32_t gu_tmem_cols() { return 2 * NQ <= 32 ? 32 : (2 * NQ <= 64 ? 64 : 128); }

template <int NQ>
__host__ __device__ constexpr size_t gu_smem_bytes() {
  return 1024 + (size_t)GU_NS * gu_stage_bytes<NQ>() + 8 * (2 * GU_NS + 4) + 16;
}

// three BF16 slices of a pair of FP32 values (stored as bf16x2 words)
__device__ __forceinline__ void split3(float x, float y, __nv_bfloat162& s0, __nv_bfloat162& s1,
                                       __nv_bfloat162& s2) {
  s0 = __floats2bfloat162_rn(x, y);
  const float2 f0 = __bfloat1622float2(s0);
  const float rx = x - f0.x, ry = y - f0.y;
  s1 = __floats2bfloat162_rn(rx, ry);
  const float2 f1 = __bfloat1622float2(s1);
  s2 = __floats2bfloat162_rn(rx - f1.x, ry - f1.y);
}

// part[blk][tile][GU_M][NQ]: the block's FP64 sums of its rows
template <int NQ>
__global__ void __launch_bounds__(GU_THREADS, 1)
    k_gram_umma(int64_t N, int p, int q, const float* __restrict__ A, int64_t lda, const float* __restrict__ B,
                int64_t ldb, int64_t rows_per_blk, double* __restrict__ part, int* __restrict__ err) {
  constexpr int SB = gu_stage_bytes<NQ>();
  constexpr int B_SLICE = NQ * 128;
  constexpr int NA = GU_M / GU_WARPS, NB = NQ / GU_WARPS;   // A and B columns per warp
  constexpr int NH = NQ / 2;          // C columns per drain warp
  constexpr uint32_t TCOLS = gu_tmem_cols<NQ>();
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + (size_t)GU_NS * SB);
  uint64_t* full = bars;                     // [GU_NS] operands of a stage stored
  uint64_t* mma_done = bars + GU_NS;         // [GU_NS] and read
  uint64_t* acc_full = bars + 2 * GU_NS;     // [2]
  uint64_t* acc_empty = acc_full + 2;        // [2]
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * GU_M;
  const int64_t r_begin = blockIdx.x * rows_per_blk;
  const int64_t r_end = min(N, r_begin + rows_per_blk);
  const int nch = r_begin < r_end ? (int)((r_end - r_begin + GU_K - 1) / GU_K) : 0;

  if (tid == 0) {
    for (int i = 0; i < GU_NS; ++i) {
      mbar_init(&full[i], GU_WARPS);
      mbar_init(&mma_done[i], 1u);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1u);
      mbar_init(&acc_empty[i], 8u);
    }
  }
  if (warp == 0) tmem_alloc(tmem_holder, TCOLS);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tacc = *tmem_holder;

  const int ngrp = (nch + GU_F - 1) / GU_F;
  if (warp < GU_WARPS) {
    // ------------------------------------------------------------ producers
    // this thread's columns: A columns m0 + warp + 16u, B columns warp + 16u;
    // rows r0 + 2 lane, r0 + 2 lane + 1 of each stage
    // (only the A columns below p: the other rows of the operand tile, whatever
    // they hold, feed output rows that nothing reads)
    const int nu = min(NA, (p - m0 - warp + GU_WARPS - 1) / GU_WARPS);
    const float* const colA = A + (int64_t)(m0 + warp) * lda + r_begin + 2 * lane;
    const float* const colB = B + (int64_t)warp * ldb + r_begin + 2 * lane;
    const int64_t nrow = r_end - r_begin;
    // 8-byte loads where every column allows them (r_begin is a multiple of 64)
    const bool pairs = ((lda | ldb) & 1) == 0 && (((uintptr_t)A | (uintptr_t)B) & 7) == 0;
    struct Stage {
      float2 a[NA], b[NB];
    };
    auto fetch = [&](int i, Stage& x) {
      const int64_t o = (int64_t)i * GU_K;
      const float* pa = colA + o;
      const float* pb = colB + o;
      const bool ok0 = o + 2 * lane < nrow, ok1 = o + 2 * lane + 1 < nrow;
#pragma unroll
      for (int u = 0; u < NA; ++u, pa += GU_WARPS * lda) {
        if (u >= nu) break;
        if (pairs && ok1) {
          x.a[u] = __ldg(reinterpret_cast<const float2*>(pa));
        } else {
          x.a[u].x = ok0 ? __ldg(pa) : 0.f;
          x.a[u].y = ok1 ? __ldg(pa + 1) : 0.f;
        }
      }
#pragma unroll
      for (int u = 0; u < NB; ++u, pb += GU_WARPS * ldb) {
        const bool in = warp + GU_WARPS * u < q;
        if (pairs && ok1 && in) {
          x.b[u] = __ldg(reinterpret_cast<const float2*>(pb));
        } else {
          x.b[u].x = in && ok0 ? __ldg(pb) : 0.f;
          x.b[u].y = in && ok1 ? __ldg(pb + 1) : 0.f;
        }
      }
    };
    auto put = [&](unsigned char* at, int slice, const float2& x) {
      __nv_bfloat162 s0, s1, s2;
      split3(x.x, x.y, s0, s1, s2);
      *reinterpret_cast<__nv_bfloat162*>(at) = s0;
      *reinterpret_cast<__nv_bfloat162*>(at + slice) = s1;
      *reinterpret_cast<__nv_bfloat162*>(at + 2 * slice) = s2;
    };
    // one stage: P holds its values, and those two stages on afterwards
    auto step = [&](int i, Stage& P) -> bool {
      const int s = i % GU_NS;
      if (!mbar_wait_warp(&mma_done[s], ((uint32_t)(i / GU_NS) & 1u) ^ 1u, err, 1)) return false;
      unsigned char* sa = base + (size_t)s * SB;
#pragma unroll
      for (int u = 0; u < NA; ++u) {
        if (u >= nu) break;
        put(sa + sw128_off(warp + GU_WARPS * u, 2 * lane), GU_A_SLICE, P.a[u]);
      }
#pragma unroll
      for (int u = 0; u < NB; ++u)
        put(sa + 3 * GU_A_SLICE + sw128_off(warp + GU_WARPS * u, 2 * lane), B_SLICE, P.b[u]);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[s]);
      if (i + 2 < nch) fetch(i + 2, P);
      return true;
    };
    Stage even, odd;
    if (nch > 0) fetch(0, even);
    if (nch > 1) fetch(1, odd);
    for (int i = 0; i < nch; i += 2) {
      if (!step(i, even)) break;
      if (i + 1 < nch && !step(i + 1, odd)) break;
    }
  } else if (warp < GU_WARPS + 8) {
    // --------------------------------------------------------------- drains
    // double-float sums of row 32 (warp & 3) + lane (its TMEM lane) of C
    const int half = (warp - GU_WARPS) >> 2;
    df acc[NH];
#pragma unroll
    for (int j = 0; j < NH; ++j) acc[j] = df{0.f, 0.f};
    const uint32_t at = tacc + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(half * NH);
    for (int grp = 0; grp < ngrp; ++grp) {
      const int ab = grp & 1;
      if (!mbar_wait_warp(&acc_full[ab], (uint32_t)(grp >> 1) & 1u, err, 3)) break;
      fence_after_sync();
      float v[NH];
#pragma unroll
      for (int j0 = 0; j0 < NH; j0 += 8) tmem_ld8(at + (uint32_t)(ab * NQ + j0), *reinterpret_cast<float(*)[8]>(v + j0));
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[ab]);
#pragma unroll
      for (int j = 0; j < NH; ++j) acc[j] = df_add(acc[j], df{v[j], 0.f});
    }
    double* out = part + ((int64_t)blockIdx.x * gridDim.y + blockIdx.y) * (GU_M * NQ) +
                  (int64_t)(32 * (warp & 3) + lane) * NQ + half * NH;
#pragma unroll
    for (int j = 0; j < NH; ++j) out[j] = df_value(acc[j]);
  } else {
    // ----------------------------------------------------------- MMA issuer
    constexpr uint64_t KMAJ = sdesc(0, 16, 1024, LAYOUT_SW128);
    constexpr uint32_t idesc = idesc_bf16(GU_M, NQ, 0, 0);
    constexpr int PA[6] = {0, 0, 1, 0, 1, 2}, PB[6] = {0, 1, 0, 2, 1, 0};
    int issued = 0;
    for (int i = 0; i < nch; ++i) {
      const int s = i % GU_NS, grp = i / GU_F, ab = grp & 1;
      bool ok = true;
      if (i % GU_F == 0) ok = mbar_wait_warp(&acc_empty[ab], ((uint32_t)(grp >> 1) & 1u) ^ 1u, err, 2);
      ok = ok && mbar_wait_warp(&full[s], (uint32_t)(i / GU_NS) & 1u, err, 5);
      if (!ok) break;
      fence_after_sync();
      const uint64_t ad = KMAJ + (smem_u32(base + (size_t)s * SB) >> 4), bd = ad + 3 * GU_A_SLICE / 16;
      const uint32_t d = tacc + (uint32_t)(ab * NQ);
      if (elect_one()) {
        mma_bf16(d, ad, bd, idesc, (i % GU_F) ? 1u : 0u);
#pragma unroll
        for (int pr = 0; pr < 6; ++pr)
#pragma unroll
          for (int ks = pr == 0 ? 1 : 0; ks < GU_K / 16; ++ks)
            mma_bf16_c<true>(d, ad + PA[pr] * (GU_A_SLICE / 16) + 2 * ks, bd + PB[pr] * (B_SLICE / 16) + 2 * ks, idesc);
        mma_commit(&mma_done[s]);
        if (i % GU_F == GU_F - 1 || i == nch - 1) mma_commit(&acc_full[ab]);
      }
      __syncwarp();
      issued = i + 1;
    }
    // no MMA may still be running when TMEM is released: wait (bounded) for
    // the last commit of every stage
    for (int k = 0; k < GU_NS && k < issued; ++k) {
      const int i = issued - 1 - k;
      mbar_wait_warp(&mma_done[i % GU_NS], (uint32_t)(i / GU_NS) & 1u, err, 4);
    }
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  if (warp == 0) {
    tmem_dealloc(tacc, TCOLS);
    tmem_relinquish();
  }
}

// C(p x q) (col-major, ldc) = alpha * sum over blocks (fixed order) + beta C;
// one warp per output (one thread each took 54 us for 50 x 20 outputs)
__global__ void __launch_bounds__(256) k_gram_umma_reduce(int p, int q, int nq, int nblk, int ntile,
                                                          const double* __restrict__ part, double* __restrict__ C,
                                                          int ldc, double alpha, double beta) {
  const int lane = threadIdx.x & 31;
  for (int o = (blockIdx.x * 256 + threadIdx.x) >> 5; o < p * q; o += gridDim.x * 8) {
    const int i = o / q, j = o - i * q;
    const int tile = i / GU_M, ii = i - tile * GU_M;
    double s = 0.0;
    for (int b = lane; b < nblk; b += 32) s += part[((int64_t)b * ntile + tile) * (GU_M * nq) + (int64_t)ii * nq + j];
#pragma unroll
    for (int t = 16; t; t >>= 1) s += __shfl_xor_sync(0xffffffffu, s, t);
    if (lane == 0) {
      const double prev = beta == 0.0 ? 0.0 : beta * C[(int64_t)j * ldc + i];
      C[(int64_t)j * ldc + i] = prev + alpha * s;
    }
  }
}

}  // namespace

struct GramPlan {
  int* d_err = nullptr;
  int* h_err = nullptr;
  int off = 0;                  // 1: the CUDA-core kernel is used instead
};

void gram_free(Ctx* c) {
  GramPlan* g = reinterpret_cast<GramPlan*>(c->gram);
  if (!g) return;
  dfree(c, g->d_err);
  if (g->h_err) cudaFreeHost(g->h_err);
  delete g;
  c->gram = nullptr;
}

int gram_set_off(Ctx* c, int off) {
  if (!c->gram) c->gram = new GramPlan;
  reinterpret_cast<GramPlan*>(c->gram)->off = off;
  return ADCGPU_OK;
}

bool gram_umma_usable(Ctx* c, int64_t N, int p, int q) {
  if (q < 1 || q > 48 || p < 1 || N < 1) return false;
  if (c->gram && reinterpret_cast<GramPlan*>(c->gram)->off) return false;
  int major = 0;
  if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, c->device) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return major >= 10 && gu_smem_bytes<48>() <= (size_t)smem_optin_max(c);
}

int gram_umma(Ctx* c, Workspace& ws, int64_t N, int p, int q, const float* A, int64_t lda, const float* B,
              int64_t ldb, double* C, int ldc, double alpha, double beta) {
  if (!c->gram) c->gram = new GramPlan;
  GramPlan* gp = reinterpret_cast<GramPlan*>(c->gram);
  if (!gp->d_err) {
    ST(dmalloc(c, (void**)&gp->d_err, sizeof(int)));
    ADC_CUDA(c, cudaMallocHost((void**)&gp->h_err, sizeof(int)));
    ADC_CUDA(c, cudaMemsetAsync(gp->d_err, 0, sizeof(int), c->stream));
  }
  const int nq = q <= 16 ? 16 : (q <= 32 ? 32 : 48);
  const int ntile = (p + GU_M - 1) / GU_M;
  // one block per SM over all column tiles (one fits an SM), each row block a
  // multiple of the stage height
  const int64_t want = std::max<int64_t>(1, (int64_t)c->nsm / ntile);
  const int64_t rows = std::max<int64_t>(GU_K, ((N + want - 1) / want + GU_K - 1) / GU_K * GU_K);
  const int nblk = (int)((N + rows - 1) / rows);
  ST(ws.reserve(c, sizeof(double) * (size_t)nblk * ntile * GU_M * nq));
  double* part = reinterpret_cast<double*>(ws.p);
  const int smax = smem_optin_max(c);
  auto go = [&](auto kern, size_t smem) -> int {
    ADC_CUDA(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smax));
    kern<<<dim3(nblk, ntile), GU_THREADS, smem, c->stream>>>(N, p, q, A, lda, B, ldb, rows, part, gp->d_err);
    ADC_COUNT_LAUNCH();
    ADC_CUDA(c, cudaGetLastError());
    return ADCGPU_OK;
  };
  if (nq == 16) ST(go(k_gram_umma<16>, gu_smem_bytes<16>()));
  else if (nq == 32) ST(go(k_gram_umma<32>, gu_smem_bytes<32>()));
  else ST(go(k_gram_umma<48>, gu_smem_bytes<48>()));
  k_gram_umma_reduce<<<std::min((p * q + 7) / 8, c->nsm * 8), 256, 0, c->stream>>>(p, q, nq, nblk, ntile, part,
                                                                                      C, ldc, alpha, beta);
  ADC_COUNT_LAUNCH();
  ADC_CUDA(c, cudaGetLastError());
  // the error word of the bounded waits (one small copy; the callers read C
  // on the host right after)
  ADC_CUDA(c, cudaMemcpyAsync(gp->h_err, gp->d_err, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  ADC_CUDA(c, cudaStreamSynchronize(c->stream));
  if (*gp->h_err) {
    const int code = *gp->h_err;
    ADC_CUDA(c, cudaMemsetAsync(gp->d_err, 0, sizeof(int), c->stream));
    return set_err(c, ADCGPU_DEVICE_TIMEOUT, "tensor-core Gram product: a pipeline wait timed out (stage " +
                                                  std::to_string(code) + ")");
  }
  return ADCGPU_OK;
}

}  // namespace adcgpu

using namespace adcgpu;

extern "C" int adcgpu_gram_f32(adcgpu_ctx* h, int64_t N, int p, int q, const void* dA, int64_t lda, const void* dB,
                               int64_t ldb, double* dC, int ldc) {
  Ctx* c = reinterpret_cast<Ctx*>(h);
  if (!c || N < 1 || p < 1 || q < 1 || !dA || !dB || !dC || lda < N || ldb < N || ldc < p) return ADCGPU_BAD_INPUT;
  cudaSetDevice(c->device);
  Workspace ws;
  int st = gemm_tn<float, double, double>(c, ws, N, p, q, (const float*)dA, lda, (const float*)dB, ldb, dC, ldc, 1.0,
                                          0.0);
  if (st) return st;
  ADC_CUDA(c, cudaStreamSynchronize(c->stream));
  return ADCGPU_OK;
}
