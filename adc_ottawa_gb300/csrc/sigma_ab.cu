// Segments A and B of the coupling block (the singles (a', k) and (b', k) of
// a double (a', b', k', l'); layout in internal.h) for the mixed-precision
// sigma product: BF16 values by mma.sync runs (k_seg_bf16), FP32 values beside
// the CUDA-core tile or the two-pass tcgen05 product in compact form.  Replaces the per-(slab, b') pass 2 and the
// per-run pass 3 of sigma.cu on the BF16 tensor-core path and the FP32-value
// tiled path; the product is that of hxvec_incore (block_davidson.f90:
// 844-883) restricted to these entries.
//
// The compact form.  In a slab of a class with a' < b' (classes 2, 4I, 4II,
// fixed k', l') the segment-A entry of row (a', b') at a hole k outside
// {k', l'} is the coupling of (a', k) with the double, and the coincidence
// tests of C1, C2 and C4_ph_2p2h (adc_ph.f90:974-1054) leave only the term
// that depends on (b', k, k', l'): the same FP64 value, thresholded the same
// way, for every a'.  Likewise the segment-B entry depends on (a', k) only.
// So per slab
//     segA[(a',b'), k] = Y[b', k] + [k = k'] P(a',b') + [k = l'] Q(a',b')
//     segB[(a',b'), k] = Z[a', k] + [k = k'] R(a',b') + [k = l'] S(a',b')
// with Y, Z zero at k', l' and P, Q, R, S the stored coincident entries
// (Q = S = 0 when k' = l').  The tables are copied out of the value store, so
// they reproduce it exactly.  With them the slab's products are small dense
// contractions over k (16 values) and over a' or b', and the rows are read
// in storage order:
//   W2[(a',b'), c] += sum_k segA[k] V[(a',k), c] + sum_k segB[k] V[(b',k), c]
//   W1[(b',k), c]  += sum_{a'<b'} segB[(a',b'), k] V2[(a',b'), c]     (phase 1)
//   W1[(a',k), c]  += sum_{b'>a'} segA[(a',b'), k] V2[(a',b'), c]     (phase 2)
// Rows of the classes with a' = b' (1 and 3) carry segment A only and are
// handled row by row by k_ab_diag.
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "internal.h"

namespace adcgpu {

namespace {

// slab s of the classes with a' < b': s < no -> class 2 (k' = l' = s);
// otherwise classes 4I / 4II, hole pair s - no (mod npair_o)
struct PairSlab {
  int cls, kp, lp;
  int64_t row0;
};

__host__ __device__ inline PairSlab pair_slab(const GeomDev& g, int s) {
  PairSlab r;
  if (s < g.no) {
    r.cls = 1; r.kp = r.lp = s;
    r.row0 = g.start[1] + (int64_t)s * g.npair_v;
  } else {
    const int64_t t = s - g.no;
    r.cls = 3 + (int)(t / g.npair_o);
    const int64_t p = t % g.npair_o;
    pair_decode(p, g.no, r.kp, r.lp);
    r.row0 = g.start[r.cls] + p * g.npair_v;
  }
  return r;
}

// index of a pair-class row in the coincident-entry table
__host__ __device__ inline int64_t pair_row_index(const GeomDev& g, int cls, int64_t row) {
  return cls == 1 ? row - g.start[1] : (g.start[2] - g.start[1]) + (row - g.start[3]);
}

template <typename TV> __device__ inline float to_f(TV x);
template <> __device__ inline float to_f<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <> __device__ inline float to_f<float>(float x) { return x; }

// Copies Y, Z and the coincident entries out of the value store.
__global__ void k_ab_extract(GeomDev g, const float* __restrict__ Bt, int nslab, float* __restrict__ Y,
                             float* __restrict__ Z, float4* __restrict__ coin) {
  const int nv = g.nv, no = g.no, noP = g.noP;
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nth = (int64_t)gridDim.x * blockDim.x;
  // Y[s][b][k], Z[s][a][k]
  const int64_t ntab = (int64_t)nslab * nv * noP;
  for (int64_t i = tid; i < ntab; i += nth) {
    const int k = (int)(i % noP);
    const int x = (int)((i / noP) % nv);
    const int s = (int)(i / ((int64_t)noP * nv));
    const PairSlab ps = pair_slab(g, s);
    const int64_t L = g.len[ps.cls];
    const bool kin = k < no && k != ps.kp && k != ps.lp;
    float y = 0.f, z = 0.f;
    if (kin && x >= 1) {           // row (0, x): segment A at k
      const int64_t row = ps.row0 + pair_index(0, x, nv);
      y = Bt[g.off[ps.cls] + (row - g.start[ps.cls]) * L + k];
    }
    if (kin && x <= nv - 2) {      // row (x, nv - 1): segment B at k
      const int64_t row = ps.row0 + pair_index(x, nv - 1, nv);
      z = Bt[g.off[ps.cls] + (row - g.start[ps.cls]) * L + noP + k];
    }
    Y[i] = y;
    Z[i] = z;
  }
  // coincident entries of every pair-class row
  const int64_t c2 = g.start[2] - g.start[1], nrow = c2 + (g.start[5] - g.start[3]);
  for (int64_t t = tid; t < nrow; t += nth) {
    const int64_t row = t < c2 ? g.start[1] + t : g.start[3] + (t - c2);
    const int cls = t < c2 ? 1 : (row < g.start[4] ? 3 : 4);
    const int64_t L = g.len[cls];
    const int64_t rl = row - g.start[cls];
    int kp, lp;
    if (cls == 1) {
      kp = lp = (int)(rl / g.npair_v);
    } else {
      pair_decode(rl / g.npair_v, no, kp, lp);
    }
    const float* rp = Bt + g.off[cls] + rl * L;
    float4 q;
    q.x = rp[kp];
    q.y = kp != lp ? rp[lp] : 0.f;
    q.z = rp[noP + kp];
    q.w = kp != lp ? rp[noP + lp] : 0.f;
    coin[t] = q;
  }
}

// swizzled 16-byte slot of (b, k) in the V1 table: the 8 lanes of a
// quarter-warp with consecutive b read 8 different bank groups
__device__ __forceinline__ int v1_slot(int b, int k, int NOPv) { return b * NOPv + (k ^ (b & 7)); }

// One CTA per (pair-class slab, 4 columns); thread b <-> virtual b.
// Phase 1 (every a' < b): W2 of row (a', b) and, in registers, the segment-B
// sums of single (b, k).  Phase 2 (DO_A; thread a): the segment-A sums of
// single (a, k) over its run of rows (a, a+1 .. nv-1).  Dynamic shared
// memory: V1 of the block's columns [nvS][NOP] float4, Z [nv][NOP], Y [NOP][nvS].
template <int NOP, bool DO_A>
__global__ void __launch_bounds__(256) k_ab_pairs(GeomDev g, const float* __restrict__ Yt,
                                                  const float* __restrict__ Zt, const float4* __restrict__ coin,
                                                  const float* __restrict__ V, int64_t ldv, int m,
                                                  float* __restrict__ W, int64_t ldw, double* __restrict__ W1,
                                                  int64_t ld1) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int nv = g.nv, no = g.no;
  const int nvS = blockDim.x;
  float4* sV1 = reinterpret_cast<float4*>(smem);
  float* sZ = reinterpret_cast<float*>(sV1 + (size_t)nvS * NOP);
  float* sY = sZ + (size_t)nv * NOP;
  const int s = blockIdx.x;
  const int c0 = blockIdx.y * 4;
  const int ncol = min(4, m - c0);
  const PairSlab ps = pair_slab(g, s);
  const int64_t n1 = g.n1;
  const int tid = threadIdx.x;
  // phase 0: tables of this slab and V1 of the four columns
  for (int i = tid; i < nv * NOP; i += nvS) {
    const int b = i / NOP, k = i - b * NOP;
    float4 v;
    float* pv = reinterpret_cast<float*>(&v);
#pragma unroll
    for (int c = 0; c < 4; ++c)
      pv[c] = (k < no && c < ncol) ? V[(int64_t)(c0 + c) * ldv + (int64_t)b * no + k] : 0.f;
    sV1[v1_slot(b, k, NOP)] = v;
    sZ[i] = Zt[((int64_t)s * nv) * NOP + i];
    if (DO_A) sY[k * nvS + b] = Yt[((int64_t)s * nv) * NOP + i];
  }
  __syncthreads();
  const int kp = ps.kp, lp = ps.lp;
  const int cls = ps.cls;
  const bool cls2 = cls == 1;
  // ------------------------------------------------------------- phase 1
  {
    const int b = tid;
    const bool act = b < nv && b >= 1;
    float accB[NOP][4];
#pragma unroll
    for (int k = 0; k < NOP; ++k)
#pragma unroll
      for (int c = 0; c < 4; ++c) accB[k][c] = 0.f;
    float accR[4] = {0.f, 0.f, 0.f, 0.f}, accS[4] = {0.f, 0.f, 0.f, 0.f};
    const int amax = act ? b : 0;
    for (int a = 0; a < amax; ++a) {
      const int64_t pr = pair_index(a, b, nv);
      const int64_t row = ps.row0 + pr;
      const int64_t d = cls2 ? g.start[1] + pr * no + kp : row;
      const float4 q = coin[pair_row_index(g, cls, row)];
      float v2[4], w2[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        v2[c] = c < ncol ? V[(int64_t)(c0 + c) * ldv + n1 + d] : 0.f;
        w2[c] = c < ncol ? W[(int64_t)(c0 + c) * ldw + n1 + d] : 0.f;
      }
      // sum_k segA[k] V1[(a,k)] + sum_k segB[k] V1[(b,k)]
#pragma unroll
      for (int k = 0; k < NOP; ++k) {
        const float zk = sZ[a * NOP + k];
        const float4 xb = sV1[v1_slot(b, k, NOP)];
        w2[0] = fmaf(zk, xb.x, w2[0]);
        w2[1] = fmaf(zk, xb.y, w2[1]);
        w2[2] = fmaf(zk, xb.z, w2[2]);
        w2[3] = fmaf(zk, xb.w, w2[3]);
        if (DO_A) {
          const float yk = sY[k * nvS + b];              // consecutive b: no bank conflicts
          const float4 xa = sV1[v1_slot(a, k, NOP)];   // the same for the whole CTA: broadcast
          w2[0] = fmaf(yk, xa.x, w2[0]);
          w2[1] = fmaf(yk, xa.y, w2[1]);
          w2[2] = fmaf(yk, xa.z, w2[2]);
          w2[3] = fmaf(yk, xa.w, w2[3]);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) accB[k][c] = fmaf(zk, v2[c], accB[k][c]);
      }
      // coincident entries
      {
        const float4 bk = sV1[v1_slot(b, kp, NOP)], bl = sV1[v1_slot(b, lp, NOP)];
        const float* pbk = reinterpret_cast<const float*>(&bk);
        const float* pbl = reinterpret_cast<const float*>(&bl);
#pragma unroll
        for (int c = 0; c < 4; ++c) w2[c] = fmaf(q.z, pbk[c], fmaf(q.w, pbl[c], w2[c]));
        if (DO_A) {
          const float4 ak = sV1[v1_slot(a, kp, NOP)], al = sV1[v1_slot(a, lp, NOP)];
          const float* pak = reinterpret_cast<const float*>(&ak);
          const float* pal = reinterpret_cast<const float*>(&al);
#pragma unroll
          for (int c = 0; c < 4; ++c) w2[c] = fmaf(q.x, pak[c], fmaf(q.y, pal[c], w2[c]));
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          accR[c] = fmaf(q.z, v2[c], accR[c]);
          accS[c] = fmaf(q.w, v2[c], accS[c]);
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (c < ncol) W[(int64_t)(c0 + c) * ldw + n1 + d] = w2[c];
    }
    if (act) {
#pragma unroll
      for (int k = 0; k < NOP; ++k) {
        if (k >= no) break;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c >= ncol) break;
          const float v = accB[k][c] + (k == kp ? accR[c] : 0.f) + (k == lp ? accS[c] : 0.f);
          if (v != 0.f) atomicAdd(&W1[(int64_t)(c0 + c) * ld1 + (int64_t)b * no + k], (double)v);
        }
      }
    }
  }
  if (!DO_A) return;
  // ------------------------------------------------------------- phase 2
  {
    const int a = tid;
    if (a >= nv - 1) return;
    float acc[NOP][4];
#pragma unroll
    for (int k = 0; k < NOP; ++k)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[k][c] = 0.f;
    float accP[4] = {0.f, 0.f, 0.f, 0.f}, accQ[4] = {0.f, 0.f, 0.f, 0.f};
    const int64_t pr0 = pair_index(a, a + 1, nv);
    for (int b = a + 1; b < nv; ++b) {
      const int64_t pr = pr0 + (b - a - 1);
      const int64_t row = ps.row0 + pr;
      const int64_t d = cls2 ? g.start[1] + pr * no + kp : row;
      const float4 q = coin[pair_row_index(g, cls, row)];
      float v2[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) v2[c] = c < ncol ? V[(int64_t)(c0 + c) * ldv + n1 + d] : 0.f;
#pragma unroll
      for (int k = 0; k < NOP; ++k) {
        const float yk = sY[k * nvS + b];
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[k][c] = fmaf(yk, v2[c], acc[k][c]);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        accP[c] = fmaf(q.x, v2[c], accP[c]);
        accQ[c] = fmaf(q.y, v2[c], accQ[c]);
      }
    }
#pragma unroll
    for (int k = 0; k < NOP; ++k) {
      if (k >= no) break;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (c >= ncol) break;
        const float v = acc[k][c] + (k == kp ? accP[c] : 0.f) + (k == lp ? accQ[c] : 0.f);
        if (v != 0.f) atomicAdd(&W1[(int64_t)(c0 + c) * ld1 + (int64_t)a * no + k], (double)v);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// BF16 values: the pair-class rows' segments on mma.sync.  A run (the rows of
// one slab with equal a', segment A, or equal b', segment B) couples to the
// singles (f, k) of its fixed virtual f:
//   W2[r, c] += sum_k R[r, k] V[(f, k), c],   W1[(f, k), c] += sum_r R[r, k] V2[r, c]
// A block takes eight consecutive f (one warp and run each) and 16 columns, 16
// rows of every run a step: their V2 and W2 entries, contiguous along a' or b'
// for the block but not for one run, move through shared memory (with a warp
// on its own, each 4-byte access of segment B was a sector of its own: 2.4 ms
// instead of 1.0).  The values come by cp.async, the next V2 and this step's
// W2 are loaded a step ahead.  The values are BF16 already; a vector entry is
// three BF16 slices, which hold its 24 bits, so the products are those of the
// FP32 vectors.  A step's sums (48 products an entry) come from one FP32
// accumulator chain, lowest slice first, and are added to the run's in FP32.
// Bound by the latency of its loads: 0.93 ms (A) and 0.96 ms (B) for 40 columns
// at nocc=16/nvirt=180, where the per-thread compact kernel above took 3.06 ms.
// ---------------------------------------------------------------------------
// segments of the pair-class rows, packed: [pair row][A, B][kw]
__global__ void k_seg_pack(GeomDev g, const __nv_bfloat16* __restrict__ Bt, int kw, __nv_bfloat16* __restrict__ out) {
  const int64_t c2 = g.start[2] - g.start[1], n = (c2 + (g.start[5] - g.start[3])) * 2 * kw;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = i / (2 * kw);
    const int x = (int)(i - t * (2 * kw)), seg = x >= kw ? 1 : 0, k = x - seg * kw;
    const int64_t row = t < c2 ? g.start[1] + t : g.start[3] + (t - c2);
    const int cls = t < c2 ? 1 : (row < g.start[4] ? 3 : 4);
    out[i] = k < g.no ? Bt[g.off[cls] + (row - g.start[cls]) * g.len[cls] + seg * g.noP + k] : __float2bfloat16(0.f);
  }
}

__device__ __forceinline__ void seg_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// three BF16 slices of a pair of FP32 values (x = s0 + s1 + s2 to 24 bits)
__device__ __forceinline__ void seg_split(float x, float y, uint32_t (&s)[3]) {
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    s[t] = *reinterpret_cast<const uint32_t*>(&h);
    x -= __low2float(h);
    y -= __high2float(h);
  }
}
// A fragments of m16n8k16: rows (columns c) lane / 4 and + 8, positions
// 2 (lane % 4), + 1, + 8, + 9
__device__ __forceinline__ void seg_frag(const float (&x)[2][4], uint32_t (&f)[3][4]) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      uint32_t s[3];
      seg_split(x[h][2 * v], x[h][2 * v + 1], s);
#pragma unroll
      for (int t = 0; t < 3; ++t) f[t][2 * v + h] = s[t];
    }
}

constexpr int SEG_F = 8;
template <bool SEGB>
__global__ void __launch_bounds__(32 * SEG_F)
    k_seg_bf16(GeomDev g, int nslab, int ngrp, const __nv_bfloat16* __restrict__ seg, const float* __restrict__ V,
                 int64_t ldv, int m, float* __restrict__ W, int64_t ldw, double* __restrict__ W1, int64_t ld1) {
  constexpr int KT = 1;   // k tiles of 16 holes: the pass takes nocc <= 16
  constexpr int PITCH = KT * 32 + 16, KW = 16 * KT, NPIECE = 32 * KT;
  constexpr int PA = SEG_F + 1, PC = 16 * PA + 1;        // pitches of a' and c in the tiles
  __shared__ __align__(16) unsigned char smem_seg[SEG_F * 2 * 16 * PITCH];
  __shared__ float sV[16 * PC], sW[16 * PC];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem_seg + wid * 2 * 16 * PITCH);
  const int no = g.no, nv = g.nv;
  const int64_t n1 = g.n1;
  const int pos[4] = {2 * tig, 2 * tig + 1, 2 * tig + 8, 2 * tig + 9};
  // this thread's part of a tile: fixed virtual f0 + tb, the other o0 + ta,
  // columns tc + 2 j; consecutive threads along b'
  const int tb = SEGB ? tid & 7 : (tid >> 4) & 7, ta = SEGB ? (tid >> 3) & 15 : tid & 15, tc = tid >> 7;
  const int nfb = (nv - 1 + SEG_F - 1) / SEG_F;
  const int64_t nblk = (int64_t)nslab * ngrp * nfb;
  for (int64_t blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
    const int f0 = (SEGB ? 1 : 0) + SEG_F * (int)(blk % nfb);
    const int64_t sg = blk / nfb;
    const int c0 = (int)(sg % ngrp) * 16;
    const PairSlab ps = pair_slab(g, (int)(sg / ngrp));
    // this warp's run: f with every a' < f (SEGB), or every b' > f
    const int f = f0 + wid;
    const int obeg = SEGB ? 0 : f0 + 1, oend = SEGB ? min(f0 + SEG_F - 1, nv - 1) : nv;
    auto valid = [&](int fx, int o) { return SEGB ? fx < nv && o < fx : fx < nv - 1 && o > fx && o < nv; };
    auto pair_of = [&](int fx, int o) -> int64_t { return SEGB ? pair_index(o, fx, nv) : pair_index(fx, o, nv); };
    const int dstr = ps.cls == 1 ? no : 1;
    const int64_t dbase = n1 + (ps.cls == 1 ? g.start[1] + ps.kp : ps.row0);
    const __nv_bfloat16* sv = seg + (pair_row_index(g, ps.cls, ps.row0) * 2 + (SEGB ? 1 : 0)) * KW;
    auto issue = [&](int o0, int b) {
      for (int p = lane; p < NPIECE; p += 32) {
        const int rr = p / (2 * KT), w = p - rr * (2 * KT);
        const bool ok = valid(f, o0 + rr);
        const __nv_bfloat16* src = sv + (ok ? pair_of(f, o0 + rr) : 0) * 2 * KW + 8 * w;
        const int n = ok ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sbase + (uint32_t)((b * 16 + rr) * PITCH + 16 * w)),
                     "l"(src), "r"(n));
      }
      asm volatile("cp.async.commit_group;\n" ::);
    };
    issue(obeg, 0);
    float v[8], w[8];
    auto load_v = [&](int o0) {
      const bool ok = valid(f0 + tb, o0 + ta);
      const int64_t d = dbase + (ok ? pair_of(f0 + tb, o0 + ta) : 0) * dstr;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = c0 + tc + 2 * j;
        v[j] = ok && c < m ? __ldg(V + (int64_t)c * ldv + d) : 0.f;
      }
    };
    load_v(obeg);
    uint32_t xf[KT][3][4];
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
      float xk[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int k = 16 * kt + pos[u], c = c0 + gid + 8 * h;
          xk[h][u] = (f < nv && k < no && c < m) ? __ldg(V + (int64_t)c * ldv + (int64_t)f * no + k) : 0.f;
        }
      seg_frag(xk, xf[kt]);
    }
    float a1[2 * KT][4];
#pragma unroll
    for (int n = 0; n < 2 * KT; ++n) a1[n][0] = a1[n][1] = a1[n][2] = a1[n][3] = 0.f;
    int b = 0;
    for (int o0 = obeg; o0 < oend; o0 += 16, b ^= 1) {
#pragma unroll
      for (int j = 0; j < 8; ++j) sV[(tc + 2 * j) * PC + ta * PA + tb] = v[j];
      if (o0 + 16 < oend) issue(o0 + 16, b ^ 1);
      else asm volatile("cp.async.commit_group;\n" ::);
      __syncthreads();
      // this step's W2 and the next step's V2, ahead of their use
      const bool wok = valid(f0 + tb, o0 + ta);
      const int64_t wd = dbase + (wok ? pair_of(f0 + tb, o0 + ta) : 0) * dstr;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = c0 + tc + 2 * j;
        w[j] = wok && c < m ? W[(int64_t)c * ldw + wd] : 0.f;
      }
      if (o0 + 16 < oend) load_v(o0 + 16);
      float x[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int u = 0; u < 4; ++u) x[h][u] = sV[(gid + 8 * h) * PC + pos[u] * PA + wid];
      uint32_t vf[3][4];
      seg_frag(x, vf);
      asm volatile("cp.async.wait_group 1;\n" ::);
      __syncwarp();
#pragma unroll
      for (int kt = 0; kt < KT; ++kt) {
        uint32_t q[4];
        const uint32_t at = sbase + (uint32_t)((b * 16 + (lane & 15)) * PITCH + (lane >> 4) * 16 + kt * 32);
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]) : "r"(at));
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int t = 2; t >= 0; --t) seg_mma(s, vf[t], q[2 * n], q[2 * n + 1]);
#pragma unroll
          for (int i = 0; i < 4; ++i) a1[2 * kt + n][i] += s[i];
        }
      }
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t q[2 * KT];
#pragma unroll
        for (int kt = 0; kt < KT; ++kt) {
          const uint32_t at = sbase + (uint32_t)((b * 16 + 8 * hr + (lane & 7)) * PITCH + ((lane >> 3) & 1) * 16 + kt * 32);
          asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n"
                       : "=r"(q[2 * kt]), "=r"(q[2 * kt + 1]) : "r"(at));
        }
#pragma unroll
        for (int t = 2; t >= 0; --t)
#pragma unroll
          for (int kt = 0; kt < KT; ++kt) seg_mma(s, xf[kt][t], q[2 * kt], q[2 * kt + 1]);
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int h = 0; h < 2; ++h) sW[(gid + 8 * h) * PC + (8 * hr + pos[u]) * PA + wid] = s[2 * h + u];
      }
      __syncthreads();   // sW complete; sV and this stage of the values read
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = c0 + tc + 2 * j;
        if (wok && c < m) W[(int64_t)c * ldw + wd] = w[j] + sW[(tc + 2 * j) * PC + ta * PA + tb];
      }
    }
#pragma unroll
    for (int n = 0; n < 2 * KT; ++n)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int k = 8 * n + 2 * tig + u;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = c0 + gid + 8 * h;
          if (f < nv && k < no && c < m && a1[n][2 * h + u] != 0.f)
            atomicAdd(&W1[(int64_t)c * ld1 + (int64_t)f * no + k], (double)a1[n][2 * h + u]);
        }
      }
    __syncthreads();     // sW's readers, before the next block's tile
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
}

// Segment A of the rows with a' = b' (classes 1 and 3: one row per virtual a
// in each slab).  Thread <-> (a, 4 columns) over a group of per slabs
// (class-1 slabs k' = 0..no-1, then the class-3 hole pairs): V1[(a, k)] of its
// columns in registers, W2 of each row updated, the W1 sums of single (a, k)
// accumulated over the group.
template <typename TV, int NOP>
__global__ void __launch_bounds__(256) k_ab_diag(GeomDev g, const TV* __restrict__ Bt, const float* __restrict__ V,
                                                 int64_t ldv, int m, int per, float* __restrict__ W, int64_t ldw,
                                                 double* __restrict__ W1, int64_t ld1) {
  const int nv = g.nv, no = g.no;
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  const int c0 = blockIdx.y * 4;
  const int ncol = min(4, m - c0);
  if (a >= nv) return;
  const int nslab = no + (int)g.npair_o;
  const int q0 = blockIdx.z * per, q1 = min(nslab, q0 + per);
  const int64_t n1 = g.n1;
  float x1[NOP][4], acc[NOP][4];
#pragma unroll
  for (int k = 0; k < NOP; ++k)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      x1[k][c] = (k < no && c < ncol) ? V[(int64_t)(c0 + c) * ldv + (int64_t)a * no + k] : 0.f;
      acc[k][c] = 0.f;
    }
  for (int q = q0; q < q1; ++q) {
    const int cls = q < no ? 0 : 2;
    const int64_t row = q < no ? (int64_t)q * nv + a : g.start[2] + (int64_t)(q - no) * nv + a;
    const TV* rp = Bt + g.off[cls] + (row - g.start[cls]) * g.len[cls];
    float va[NOP];
#pragma unroll
    for (int k = 0; k < NOP; ++k) va[k] = to_f(rp[k]);
    float v2[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      v2[c] = c < ncol ? V[(int64_t)(c0 + c) * ldv + n1 + row] : 0.f;
      float w = 0.f;
#pragma unroll
      for (int k = 0; k < NOP; ++k) w = fmaf(va[k], x1[k][c], w);
      if (c < ncol) W[(int64_t)(c0 + c) * ldw + n1 + row] += w;
    }
#pragma unroll
    for (int k = 0; k < NOP; ++k)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[k][c] = fmaf(va[k], v2[c], acc[k][c]);
  }
#pragma unroll
  for (int k = 0; k < NOP; ++k) {
    if (k >= no) break;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (c >= ncol) break;
      if (acc[k][c] != 0.f) atomicAdd(&W1[(int64_t)(c0 + c) * ld1 + (int64_t)a * no + k], (double)acc[k][c]);
    }
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct AbTables {
  const void* made_from = nullptr;   // the value store the tables were copied from
  float* Y = nullptr;                // [nslab][nv][noP]
  float* Z = nullptr;
  float4* coin = nullptr;            // [pair-class rows]
  __nv_bfloat16* seg = nullptr;      // BF16 store: [pair-class rows][A, B][kw]
};

struct AbPlan {
  AbTables t[2];                     // 0: from the BF16 store, 1: from the FP32 store
};

bool ab_supported(const Ctx* c) {
  const Geometry& G = c->geom;
  return (G.noP == 8 || G.noP == 16 || G.noP == 24 || G.noP == 32) && G.nv >= 2 && G.nv <= 256 && G.no >= 1;
}

// The value store was rewritten (a new matrix): the tables are copied again
// on their next use.
void ab_invalidate(void* handle) {
  AbPlan* p = reinterpret_cast<AbPlan*>(handle);
  if (p)
    for (auto& t : p->t) t.made_from = nullptr;
}

void ab_free(Ctx* c, void*& handle) {
  AbPlan* p = reinterpret_cast<AbPlan*>(handle);
  if (!p) return;
  for (auto& t : p->t) {
    dfree(c, t.Y);
    dfree(c, t.Z);
    dfree(c, t.coin);
    dfree(c, t.seg);
  }
  delete p;
  handle = nullptr;
}

static int ab_tables(Ctx* c, void*& handle, int which, const void* Bt) {
  if (!handle) handle = new AbPlan;
  AbTables& t = reinterpret_cast<AbPlan*>(handle)->t[which];
  if (t.made_from == Bt && (t.Y || t.seg)) return ADCGPU_OK;
  const Geometry& G = c->geom;
  const GeomDev g = to_dev(G);
  const int nslab = G.no + 2 * (int)G.npair_o;
  const size_t ntab = (size_t)nslab * G.nv * G.noP;
  const size_t nrow = (size_t)((G.start[2] - G.start[1]) + (G.start[5] - G.start[3]));
  int st;
  if (which == 0) {
    const int kw = (G.no + 15) / 16 * 16;
    if (!t.seg && (st = dmalloc(c, (void**)&t.seg, sizeof(uint16_t) * std::max<size_t>(nrow, 1) * 2 * kw))) return st;
    k_seg_pack<<<c->nsm * 8, 256, 0, c->stream>>>(g, (const __nv_bfloat16*)Bt, kw, t.seg);
    ADC_COUNT_LAUNCH();
    ADC_CUDA(c, cudaGetLastError());
    t.made_from = Bt;
    return ADCGPU_OK;
  }
  if (!t.Y && (st = dmalloc(c, (void**)&t.Y, sizeof(float) * ntab))) return st;
  if (!t.Z && (st = dmalloc(c, (void**)&t.Z, sizeof(float) * ntab))) return st;
  if (!t.coin && (st = dmalloc(c, (void**)&t.coin, sizeof(float4) * std::max<size_t>(nrow, 1)))) return st;
  k_ab_extract<<<c->nsm * 8, 256, 0, c->stream>>>(g, (const float*)Bt, nslab, t.Y, t.Z, t.coin);
  ADC_COUNT_LAUNCH();
  ADC_CUDA(c, cudaGetLastError());
  t.made_from = Bt;
  return ADCGPU_OK;
}

// Segments A (when do_a) and B of the pair classes, and (when do_a) segment A
// of the classes with a' = b', for m columns of FP32 vectors; W2 rows are
// updated in place, the singles sums go to the FP64 accumulator W1 (ld1).
template <typename TV>
int ab_launch(Ctx* c, void*& handle, const TV* Bt, bool do_a, const float* V, int64_t ldv, int m, float* W,
              int64_t ldw, double* W1, int64_t ld1) {
  const int which = std::is_same<TV, float>::value ? 1 : 0;
  ST(ab_tables(c, handle, which, Bt));
  const AbTables& t = reinterpret_cast<AbPlan*>(handle)->t[which];
  const Geometry& G = c->geom;
  const GeomDev g = to_dev(G);
  const int nslab = G.no + 2 * (int)G.npair_o;
  const int nvS = (G.nv + 31) / 32 * 32;
  const int ncb = (m + 3) / 4;
  const size_t smem = (size_t)nvS * G.noP * 16 + (size_t)G.nv * G.noP * 4 + (do_a ? (size_t)G.noP * nvS * 4 : 0);
  // the cap is a per-function attribute shared by every host thread: set it
  // to the device maximum, not to this launch's size
  const int smax = smem_optin_max(c);
  if (smem > (size_t)smax) return set_err(c, ADCGPU_UNSUPPORTED, "segment A/B kernels: shared memory too small");
  auto pairs = [&](auto kern) -> int {
    ADC_CUDA(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smax));
    kern<<<dim3(nslab, ncb), nvS, smem, c->stream>>>(g, t.Y, t.Z, t.coin, V, ldv, m, W, ldw, W1, ld1);
    ADC_COUNT_LAUNCH();
    ADC_CUDA(c, cudaGetLastError());
    return ADCGPU_OK;
  };
  if constexpr (std::is_same<TV, __nv_bfloat16>::value) {
    const int ngrp = (m + 15) / 16;
    const int64_t nblk = (int64_t)nslab * ngrp * ((G.nv - 1 + SEG_F - 1) / SEG_F);
    const int grid = (int)std::min<int64_t>(nblk, (int64_t)c->nsm * 16);
    auto seg = [&](auto kern) -> int {
      if (nblk == 0) return ADCGPU_OK;
      kern<<<grid, 32 * SEG_F, 0, c->stream>>>(g, nslab, ngrp, t.seg, V, ldv, m, W, ldw, W1, ld1);
      ADC_COUNT_LAUNCH();
      ADC_CUDA(c, cudaGetLastError());
      return ADCGPU_OK;
    };
    // (the pass takes nocc <= 16 only, umma_supported)
    if (do_a) ST(seg(k_seg_bf16<false>));
    ST(seg(k_seg_bf16<true>));
  } else if (nslab > 0) {
    switch (G.noP) {
      case 8: ST(do_a ? pairs(k_ab_pairs<8, true>) : pairs(k_ab_pairs<8, false>)); break;
      case 16: ST(do_a ? pairs(k_ab_pairs<16, true>) : pairs(k_ab_pairs<16, false>)); break;
      case 24: ST(do_a ? pairs(k_ab_pairs<24, true>) : pairs(k_ab_pairs<24, false>)); break;
      default: ST(do_a ? pairs(k_ab_pairs<32, true>) : pairs(k_ab_pairs<32, false>)); break;
    }
  }
  if (do_a) {
    const int nq = G.no + (int)G.npair_o;
    // up to eight slabs a group (fewer atomics), fewer where that leaves SMs
    // idle (9/101, 5 columns: 12 blocks of eight slabs took 27 us)
    const int per = std::max(1, std::min(8, (G.nv + 127) / 128 * ncb * nq / (2 * c->nsm)));
    const dim3 grid((G.nv + 127) / 128, ncb, (nq + per - 1) / per);
    switch (G.noP) {
      case 8: k_ab_diag<TV, 8><<<grid, 128, 0, c->stream>>>(g, Bt, V, ldv, m, per, W, ldw, W1, ld1); break;
      case 16: k_ab_diag<TV, 16><<<grid, 128, 0, c->stream>>>(g, Bt, V, ldv, m, per, W, ldw, W1, ld1); break;
      case 24: k_ab_diag<TV, 24><<<grid, 128, 0, c->stream>>>(g, Bt, V, ldv, m, per, W, ldw, W1, ld1); break;
      default: k_ab_diag<TV, 32><<<grid, 128, 0, c->stream>>>(g, Bt, V, ldv, m, per, W, ldw, W1, ld1); break;
    }
    ADC_COUNT_LAUNCH();
    ADC_CUDA(c, cudaGetLastError());
  }
  return ADCGPU_OK;
}

template int ab_launch<__nv_bfloat16>(Ctx*, void*&, const __nv_bfloat16*, bool, const float*, int64_t, int, float*,
                                      int64_t, double*, int64_t);
template int ab_launch<float>(Ctx*, void*&, const float*, bool, const float*, int64_t, int, float*, int64_t, double*,
                              int64_t);

}  // namespace adcgpu
