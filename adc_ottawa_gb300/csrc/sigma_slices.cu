// FP64-accurate tensor-core pass of the sigma product: the C and D segments
// (the singles (a, k') and (a, l') of a double (a', b', k', l'); layout in
// internal.h) of FP64 values against FP64 vectors, or of FP32 values against
// FP32 vectors.  Replaces the CUDA-core tile (k_sigma_tile) for hxvec_incore
// (block_davidson.f90:844-883), hxq_incore (block_lanczos.f90:1325-1361) and
// matxvec_treal_incore (tdselib.f90:352-437).
//
// Exact slicing (K. Ozaki, T. Ogita, S. Oishi, S. M. Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59, 2012).  A row
// of values is scaled by a power of two to |v| < 1 and written as S base-256
// digits, v = sum_i d_i 2^(-7-8i), |d_0| <= 128, |d_i| < 256; so are the vector
// entries of a slab (one exponent per column) and of a row tile, all |d_i| <= 128.
// Every digit is an exact BF16 number, and the FP32 accumulators in TMEM add
// whole numbers.  Products of equal weight (i + j = g) share an
// accumulator; the groups g < S are kept (the dropped ones are below the last
// digit's weight) and combined with 64-bit integer arithmetic, so one
// rounding per tile replaces one per multiply-add.
//   S = 7: 55 bits below the row / column maximum (FP64 values)
//   S = 4: 31 bits (FP32 values and vectors)
// Whole sums: a group of g + 1 digit pairs reaches at most (g + 1) K 2^14 over K
// products, and FP32 adds without rounding up to 2^24.  W1 sums cover two tiles,
// K = 256 rows: g < 4 is exact whatever the digits are, and so are W2 sums of up
// to 256 values.  Longer rows (nvirt > 128) would leave the range in g = 2 and 3
// if all digits had one sign and size, so their values' digits 1 to 3 are drawn
// at random from a number's representations (d, or d - 256 and a carry), with a
// mean of at most 32, independently along rows and columns (S = 7).  Of the group
// sums that leaves the first digits' part, 2^23 at K = 512, 2^21 for each further
// digit, and a random part of standard deviation 2^14 sqrt(3 K) = 2^19.3: g < 4
// stays below 2^24 there too.  (Plain digits lost 1.2e-11 of such row sums at
// K = 512, 5e-14 at 384; tests/test_gpu_sigma_digits.py.)
// g >= 4 is whole while the partial sums stay below 2^24, which pseudo-random
// digits do by a factor of 50 (sum of n products: about 2^12 sqrt(n)); digits of
// one sign and size take it to 2^26 and lose a unit in the last of 24 bits an
// MMA, 2^-47 of their sum at most, the size of the roundings of K FP64 adds.
// S = 4: such sums lose 2^-30 of |values| |vectors|, below FP32's own rounding.
//
// What bounds it: the digit store is read once per 16 columns (S = 7), 14
// bytes per value; the tensor cores need S (S + 1) / 2 = 28 slice products.
#include <cuda_bf16.h>

#include <algorithm>
#include <string>
#include <type_traits>
#include <vector>

#include "internal.h"
#include "umma.h"

namespace adcgpu {

using namespace umma;

namespace {

constexpr int OZ_ROWS = 128;                       // rows per tile (MMA M)
constexpr int OZ_BOX = 64;                         // values per box row (128 bytes)
constexpr int OZ_SLOT_BYTES = 2 * OZ_ROWS * OZ_BOX * 2;
constexpr int OZ_EPI = 512;                        // threads of the 16 epilogue warps
constexpr int OZ_THREADS = 64 + OZ_EPI;            // and the producer and MMA issuer warps
constexpr int OZ_MAXNR = 6;                        // ring slots
constexpr int OZ_FLUSH = 2;                        // tiles per W1 accumulation in TMEM
constexpr int OZ_NONFINITE = 1 << 20;              // exponent of a column that holds inf or NaN
constexpr int OZ_EMIN = -2200;                     // below every exponent, and every sum of two
constexpr int OZ_VALUE_EMIN = -48;                 // below that of any kept value (above 1e-12)

__host__ __device__ constexpr int round16(int x) { return (x + 15) / 16 * 16; }
// Vector operands: PAD zero rows, then slice j of column c at row PAD + j NP + c.
// Value slice i multiplies the vector slices 0 .. S-1-i side by side into the
// columns of the groups i .. S-1.  With 8-column slices every other slice
// would start 8 columns off a 16-column boundary of TMEM: those start at the
// zero rows instead, one slice earlier.
template <int NP> __host__ __device__ constexpr int oz_pad() { return NP == 8 ? 8 : 0; }
template <int NP> __host__ __device__ constexpr bool oz_early(int i) { return NP == 8 && (i & 1); }
template <int S, int NP> __host__ __device__ constexpr int oz_n(int i) {   // MMA N
  return round16(NP * (S - i + (oz_early<NP>(i) ? 1 : 0)));
}
template <int NP> __host__ __device__ constexpr int oz_col(int i) { return NP * (i - (oz_early<NP>(i) ? 1 : 0)); }
template <int NP> __host__ __device__ constexpr int oz_brow(int i) { return oz_early<NP>(i) ? 0 : oz_pad<NP>(); }
// rows of a vector operand (the widest MMA reads oz_n(0) rows from oz_brow(0))
template <int S, int NP> __host__ __device__ constexpr int oz_xrows() { return oz_pad<NP>() + oz_n<S, NP>(0); }
// TMEM columns of one accumulator region: those of slice 0
template <int S, int NP> __host__ __device__ constexpr int oz_dw() { return oz_n<S, NP>(0); }

// geometry and buffering of one launch
struct OzShape {
  int nslot;        // 128-value groups of the longest C|D row
  int nb;           // buffers of D1 and of the V2 operand (1 or 2)
  int nr;           // ring slots
  uint32_t off_v2, off_ring, off_bar;   // shared-memory offsets
};

// the space the kernels work in: the stored matrix, or the CVS space (core
// holes only)
struct OzGeom {
  int no, nv, nvP;      // holes of the singles, virtuals (padded)
  int64_t n1, row0;     // singles; storage row of the first row exponent
};
// rows [row0, row1) of one slab: row r is vector element n1 + dbase + (r - row0) dstr
struct OzItem {
  int row0, row1;
  int tile;             // its first tile in the digit store, in boxes of all slices
  int holes;            // k' | l' << 8 | OZ_TWO: C and D segments | OZ_PAIRS: classes with a' < b'
  int dbase, dstr;
  int pad0, pad1;
};
constexpr int OZ_TWO = 1 << 16, OZ_PAIRS = 1 << 17;
struct OzSlab {         // pair rows (a' < b') of one slab
  int row0, dbase, dstr;
  int item0, nitem;     // its work items
  int pad0, pad1, pad2;
};

// --- digits --------------------------------------------------------------
// x = (-1)^neg m 2^(e - MB), m < 2^MB; zeros and subnormals have the smallest
// exponent, inf and NaN OZ_NONFINITE
template <typename T> struct Parts;
template <> struct Parts<double> {
  static constexpr int MB = 53;
  __device__ __forceinline__ static int exponent(double x) {
    const int f = (int)((__double2hiint(x) >> 20) & 0x7ff);
    return f == 0x7ff ? OZ_NONFINITE : max(f, 1) - 1022;
  }
  __device__ __forceinline__ static unsigned long long mantissa(double x) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    return (u & 0xfffffffffffffull) | ((u & 0x7ff0000000000000ull) ? 0x10000000000000ull : 0ull);
  }
  __device__ __forceinline__ static unsigned long long normal_mantissa(double x) {
    return ((unsigned long long)__double_as_longlong(x) & 0xfffffffffffffull) | 0x10000000000000ull;
  }
  __device__ __forceinline__ static bool neg(double x) { return __double2hiint(x) < 0; }
};
template <> struct Parts<float> {
  static constexpr int MB = 24;
  __device__ __forceinline__ static int exponent(float x) {
    const int f = (int)((__float_as_uint(x) >> 23) & 0xff);
    return f == 0xff ? OZ_NONFINITE : max(f, 1) - 126;
  }
  __device__ __forceinline__ static unsigned long long mantissa(float x) {
    const uint32_t u = __float_as_uint(x);
    return (u & 0x7fffffu) | ((u & 0x7f800000u) ? 0x800000u : 0u);
  }
  __device__ __forceinline__ static unsigned long long normal_mantissa(float x) {
    return (__float_as_uint(x) & 0x7fffffu) | 0x800000u;
  }
  __device__ __forceinline__ static bool neg(float x) { return (int)__float_as_uint(x) < 0; }
};

// balanced digits: byte i of the bias is 128
template <int S> __host__ __device__ constexpr unsigned long long oz_bias() { return S == 7 ? 0x80808080808080ull : 0x80808080ull; }
// round(x 2^(8S - 1 - h)) plus the digit bias, for x of exponent e <= h (for
// zeros too: the shift stays below the word): byte i from the top is digit i
// plus byte i of the bias
template <int S, typename T>
__device__ __forceinline__ unsigned long long oz_fixed_m(T x, unsigned long long m, int shift, unsigned long long BIAS) {
  const int e = Parts<T>::exponent(x);
  if (e == OZ_NONFINITE) return BIAS;
  const int sh = e - Parts<T>::MB + shift;
  unsigned long long q;
  if (sh >= 0) q = m << sh;
  else if (sh < -60) q = 0ull;
  else q = (m + (1ull << (-sh - 1))) >> (-sh);
  return Parts<T>::neg(x) ? BIAS - q : BIAS + q;
}
template <int S, typename T>
__device__ __forceinline__ unsigned long long oz_fixed(T x, int shift) {   // shift = 8S - 1 - h + (scale of x)
  return oz_fixed_m<S, T>(x, Parts<T>::mantissa(x), shift, oz_bias<S>());
}
// the same of a matrix value, never subnormal: zero is taken as the smallest
// normal number, far below the digits of any h >= OZ_VALUE_EMIN
template <int S, typename T>
__device__ __forceinline__ unsigned long long oz_fixed_value(T x, int shift, unsigned long long BIAS = oz_bias<S>()) {
  return oz_fixed_m<S, T>(x, Parts<T>::normal_mantissa(x), shift, BIAS);
}
// digit i as an FP32 number; its upper half is the exact BF16 one (an
// integer of at most 8 bits)
template <int S>
__device__ __forceinline__ uint32_t oz_digit(unsigned long long u, int i) {
  const uint32_t f = i == 0 ? (uint32_t)(u >> (8 * (S - 1))) : (uint32_t)(u >> (8 * (S - 1 - i))) & 0xffu;
  return __float_as_uint(__uint_as_float(0x4B000000u | f) - 8388736.0f);
}
// random biases of digits 1 to 3 of a long row's values, 32, 96, 160 or 224 (a
// digit of 256 - bias and more becomes 256 less): two random bits of the row and
// two of the position in it, combined by xor, so independent along a row and
// along a position.  Hash: splitmix64's output function (G. L. Steele, D. Lea,
// C. H. Flood, "Fast splittable pseudorandom number generators", OOPSLA 2014).
__device__ __forceinline__ unsigned long long oz_random_bits(unsigned long long x) {
  x *= 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return (x ^ (x >> 31)) & 0x00c0c0c0000000ull;
}
__device__ __forceinline__ unsigned long long oz_position_bias(int k) {
  return 0x80202020808080ull ^ oz_random_bits(2 * (unsigned long long)k + 2);
}
// digit i of a value with bias b
template <int S>
__device__ __forceinline__ uint32_t oz_digit(unsigned long long u, unsigned long long b, int i) {
  if (i == 0) return oz_digit<S>(u, 0);
  const int sh = 8 * (S - 1 - i);
  return __float_as_uint(__uint_as_float(0x4B000000u | ((uint32_t)(u >> sh) & 0xffu)) -
                         __uint_as_float(0x4B000000u | ((uint32_t)(b >> sh) & 0xffu)));
}
// two digits as a BF16 pair (lo in the lower half)
__device__ __forceinline__ uint32_t oz_pair(uint32_t lo, uint32_t hi) { return __byte_perm(lo, hi, 0x7632); }
// t 2^e of a group sum t (zero, or 2^-24 to 2^47 in size); NaN for a column
// that holds inf or NaN.  FP64: in the exponent field (the FP64 pipe takes 16
// cycles a warp for a multiplication).  A power of two outside the type's range,
// which a result inside it can need, and results at the ends of the range take
// two factors; only the second can round.
__device__ __forceinline__ double oz_pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
// (that case out of line: inlined at every result it cost the 8-column pass 2 to
// 3% of its product: 12/140, 2 columns 2632 -> 2570 us)
__device__ __noinline__ double oz_scaled_end(double t, int e) {
  if (e > (OZ_NONFINITE >> 1)) return __longlong_as_double(0x7ff8000000000000ll);
  if (t == 0.0) return t;
  e = min(max(e, -2044), 2046);
  return t * oz_pow2(e >> 1) * oz_pow2(e - (e >> 1));
}
__device__ __forceinline__ double oz_scaled(double t, int e) {
  const int hi = __double2hiint(t), f = (hi >> 20) & 0x7ff;
  if (f != 0 && (unsigned)(f + e - 1) < 2046u) return __hiloint2double(hi + (int)((unsigned)e << 20), __double2loint(t));
  return oz_scaled_end(t, e);
}
__device__ __forceinline__ float oz_scaled(float t, int e) {
  const int c = min(max(e, -252), 254), h = c >> 1;
  const float w = t * __int_as_float((h + 127) << 23) * __int_as_float((c - h + 127) << 23);
  return e > (OZ_NONFINITE >> 1) ? __int_as_float(0x7fc00000) : w;
}

// --- value digits of a range of storage rows ---------------------------------
// The digit store holds every tile of 128 rows of a slab as the shared-memory
// image the MMAs read: per 128-value group and slice two boxes of 128 rows x
// 64 values (128-byte swizzle), 32 KB in a row, so a ring slot is one
// contiguous bulk copy.  Rows past the slab's end and values past the
// segment's are zero digits.
struct OzDst {
  int64_t base[5];      // first value of the class in the digit store
  int64_t r0[5];        // first storage row of the class in the store (whole slabs)
  int64_t slab[5];      // rows of a slab
  int tps[5];           // tiles of a slab
  int nbox[5];          // 64-value boxes of a row
  int64_t tiles[6];     // tiles of the classes before this one
  int64_t row0, row1;   // storage rows [row0, row1)
};

// values between the digits of consecutive tiles of a class
template <int S> __host__ __device__ inline int64_t oz_tile_values(int nbox) { return (int64_t)S * nbox * OZ_ROWS * OZ_BOX; }

// one warp per tile row: the exponent of the largest |C|D value|, then the
// digits of 8 values per lane and step (16-byte stores, 128 bytes a box).
// Bound by HBM: 8 (4) bytes read and 2 S written per value.  LONG: geometries with
// rows of more than 256 values, whose digits 1 to 3 have random biases.
template <typename TV, int S, bool LONG>
__global__ void __launch_bounds__(256, 3) k_oz_values(GeomDev g, OzDst dst, const TV* __restrict__ Bt,
                                                   uint16_t* __restrict__ out, int16_t* __restrict__ rexp) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  __shared__ unsigned long long s_pb[LONG ? 512 : 1];
  if (LONG) {
    for (int k = threadIdx.x; k < 2 * g.nvP; k += 256) s_pb[k] = oz_position_bias(k);
    __syncthreads();
  }
  for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < dst.tiles[5] * OZ_ROWS; w += nw) {
    const int64_t tile = w / OZ_ROWS;
    const int r = (int)(w % OZ_ROWS);
    int cls = 0;
    while (cls < 4 && tile >= dst.tiles[cls + 1]) ++cls;
    const int64_t tc = tile - dst.tiles[cls];              // tile of the class
    const int64_t in_slab = tc % dst.tps[cls] * OZ_ROWS + r;
    const bool valid = in_slab < dst.slab[cls];
    const int64_t row = dst.r0[cls] + tc / dst.tps[cls] * dst.slab[cls] + in_slab;
    const bool twoa = cls == 1 || cls >= 3;
    const int nch = (cls >= 2 ? 2 : 1) * g.nvP / 8, nbox = dst.nbox[cls];
    const TV* src = Bt + g.off[cls] + (row - g.start[cls]) * g.len[cls] + (twoa ? 2 * g.noP : g.noP);
    TV v[2][8];
    int mx = OZ_VALUE_EMIN;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int q = lane + 32 * k;
#pragma unroll
      for (int u = 0; u < 8; ++u) v[k][u] = TV(0);
      if (valid && q < nch) {
        const int4* p = reinterpret_cast<const int4*>(src + 8 * q);
        int4* d = reinterpret_cast<int4*>(v[k]);
#pragma unroll
        for (int u = 0; u < (int)(8 * sizeof(TV) / 16); ++u) d[u] = __ldcs(p + u);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) mx = max(mx, Parts<TV>::exponent(v[k][u]));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    // a row that holds inf or NaN (integrals that do): its W2 entries and the
    // W1 sums of its tile become NaN
    if (lane == 0 && valid) rexp[row - dst.row0] = (int16_t)min(mx, 32767);
    uint16_t* o = out + dst.base[cls] + tc * oz_tile_values<S>(nbox);
    unsigned long long rb = 0;
    if (LONG) rb = oz_random_bits(2 * (unsigned long long)row + 1);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int q = lane + 32 * k;
      if (q >= 8 * nbox) continue;
      unsigned long long u8[8], b8[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        b8[u] = LONG && q < nch ? rb ^ s_pb[8 * q + u] : oz_bias<S>();
        u8[u] = oz_fixed_value<S, TV>(v[k][u], 8 * S - 1 - mx, b8[u]);
      }
      // 128-value group q / 16: S slices of its (one or two) boxes
      const int grp = q >> 4, bx = (q >> 3) & 1, two = 2 * grp + 1 < nbox ? 2 : 1;
      uint16_t* og = o + ((int64_t)S * 2 * grp + bx) * (OZ_ROWS * OZ_BOX) + sw128_off(r, 8 * (q & 7)) / 2;
#pragma unroll
      for (int i = 0; i < S; ++i) {
        auto pair = [&](int u) {
          if (LONG && i >= 1 && i <= 3) return oz_pair(oz_digit<S>(u8[u], b8[u], i), oz_digit<S>(u8[u + 1], b8[u + 1], i));
          return oz_pair(oz_digit<S>(u8[u], i), oz_digit<S>(u8[u + 1], i));
        };
        __stcs(reinterpret_cast<uint4*>(og + (int64_t)i * two * (OZ_ROWS * OZ_BOX)),
               make_uint4(pair(0), pair(2), pair(4), pair(6)));
      }
    }
  }
}

// Digits of the CVS matrix's pair rows (spins I, II) from its compressed
// rows: one warp per tile row spreads the kept entries over the index-free
// segments (C: (a, core hole of the slab), A: (a', k), B: (b', k)) in shared
// memory, then writes the digits of both stores as k_oz_values and
// k_oz_seg_values do.  rows: 2 npp npair (hole pair major, spin I first),
// compressed row crow0 + row.
template <int S>
__global__ void __launch_bounds__(128) k_oz_cvs_values(OzGeom g, int npp, int64_t crow0,
                                                       const int64_t* __restrict__ rowptr,
                                                       const int32_t* __restrict__ col, const double* __restrict__ val,
                                                       int kw, uint16_t* __restrict__ out, uint16_t* __restrict__ seg,
                                                       int16_t* __restrict__ rexp, int16_t* __restrict__ sexp) {
  extern __shared__ double cvs_sh[];
  const int lane = threadIdx.x & 31;
  double* row_c = cvs_sh + (threadIdx.x >> 5) * (g.nvP + 2 * kw);
  double* row_ab = row_c + g.nvP;
  const int nbox = (g.nvP + OZ_BOX - 1) / OZ_BOX;
  const int64_t npair = (int64_t)g.nv * (g.nv - 1) / 2, tps = (npair + OZ_ROWS - 1) / OZ_ROWS;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5), ntot = 2 * npp * tps * OZ_ROWS;
  for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < ntot; w += nw) {
    const int64_t tile = w / OZ_ROWS, slab = tile / tps;
    const int r = (int)(w % OZ_ROWS);
    const int64_t p = tile % tps * OZ_ROWS + r;
    const bool valid = p < npair;
    const int64_t row = slab * npair + p;
    __syncwarp();
    for (int x = lane; x < g.nvP + 2 * kw; x += 32) row_c[x] = 0.0;
    __syncwarp();
    int mc = OZ_VALUE_EMIN, ms = OZ_VALUE_EMIN;
    if (valid) {
      int ap, bp;
      pair_decode(p, g.nv, ap, bp);
      for (int64_t e = rowptr[crow0 + row] + lane; e < rowptr[crow0 + row + 1]; e += 32) {
        const int j = col[e], a = j / g.no, k = j - a * g.no;
        const double x = val[e];
        if (a == ap || a == bp) {
          row_ab[(a == bp ? kw : 0) + k] = x;
          ms = max(ms, Parts<double>::exponent(x));
        } else {
          row_c[a] = x;      // k is the slab's core hole: the row's only other couplings
          mc = max(mc, Parts<double>::exponent(x));
        }
      }
    }
    mc = __reduce_max_sync(0xffffffffu, mc);
    ms = __reduce_max_sync(0xffffffffu, ms);
    __syncwarp();
    if (lane == 0 && valid) {
      rexp[row] = (int16_t)min(mc, 32767);
      sexp[row] = (int16_t)min(ms, 32767);
    }
    uint16_t* o = out + tile * oz_tile_values<S>(nbox);
    for (int q = lane; q < 8 * nbox; q += 32) {
      unsigned long long u8[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) u8[u] = oz_fixed_value<S, double>(8 * q < g.nvP ? row_c[8 * q + u] : 0.0, 8 * S - 1 - mc);
      const int grp = q >> 4, bx = (q >> 3) & 1, two = 2 * grp + 1 < nbox ? 2 : 1;
      uint16_t* og = o + ((int64_t)S * 2 * grp + bx) * (OZ_ROWS * OZ_BOX) + sw128_off(r, 8 * (q & 7)) / 2;
#pragma unroll
      for (int i = 0; i < S; ++i)
        *reinterpret_cast<uint4*>(og + (int64_t)i * two * (OZ_ROWS * OZ_BOX)) =
            make_uint4(oz_pair(oz_digit<S>(u8[0], i), oz_digit<S>(u8[1], i)),
                       oz_pair(oz_digit<S>(u8[2], i), oz_digit<S>(u8[3], i)),
                       oz_pair(oz_digit<S>(u8[4], i), oz_digit<S>(u8[5], i)),
                       oz_pair(oz_digit<S>(u8[6], i), oz_digit<S>(u8[7], i)));
    }
    if (valid) {
      uint16_t* os = seg + row * 2 * S * kw;
      for (int x = lane; x < 2 * kw; x += 32) {
        const int sg = x >= kw ? 1 : 0, k = x - sg * kw;
        const unsigned long long u = oz_fixed_value<S, double>(row_ab[x], 8 * S - 1 - ms);
#pragma unroll
        for (int i = 0; i < S; ++i) os[(sg * S + i) * kw + k] = (uint16_t)(oz_digit<S>(u, i) >> 16);
      }
    }
  }
}

// exponents of the largest 2^rexp |V2| and 2^sexp |V2| of each work item and
// column: the scales of the V2 digits for the C|D segments (vexp) and for
// segments A and B (sexp of the classes with a' < b'; the runs of a slab take
// the maximum over its items).  One block per item and 4 columns; reads V2
// once (the pass then finds most of it in L2).
template <typename T>
__global__ void __launch_bounds__(256) k_oz_vexp(OzGeom g, const OzItem* __restrict__ items,
                                                 const int16_t* __restrict__ rexp, const int16_t* __restrict__ sexp,
                                                 const T* __restrict__ V, int64_t ldv, int m, int* __restrict__ vexp,
                                                 int* __restrict__ vsexp) {
  __shared__ int s_mx[8];
  const OzItem item = items[blockIdx.x];
  const int c0 = 4 * blockIdx.y;
  if (threadIdx.x < 8) s_mx[threadIdx.x] = OZ_EMIN;
  __syncthreads();
  int mx[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) mx[j] = OZ_EMIN;
  const bool pairs = item.holes & OZ_PAIRS;
  for (int row = item.row0 + threadIdx.x; row < item.row1; row += 256) {
    const int64_t d = item.dbase + (int64_t)(row - item.row0) * item.dstr;
    const int rx = rexp[row - g.row0], sx = pairs ? (int)sexp[row - g.row0] : OZ_EMIN;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (c0 + j >= m) break;
      const int e = Parts<T>::exponent(__ldg(V + (int64_t)(c0 + j) * ldv + g.n1 + d));
      if (e == OZ_NONFINITE || rx == 32767 || sx == 32767) mx[j] = mx[4 + j] = OZ_NONFINITE;
      else {
        mx[j] = max(mx[j], e + rx);
        mx[4 + j] = max(mx[4 + j], e + sx);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    mx[j] = __reduce_max_sync(0xffffffffu, mx[j]);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_mx[j], mx[j]);
  }
  __syncthreads();
  if (threadIdx.x < 4 && c0 + (int)threadIdx.x < m) {
    vexp[(int64_t)blockIdx.x * m + c0 + threadIdx.x] = s_mx[threadIdx.x];
    vsexp[(int64_t)blockIdx.x * m + c0 + threadIdx.x] = s_mx[4 + threadIdx.x];
  }
}

// --- the pass -----------------------------------------------------------------
enum OzBar { O_XFULL = 0, O_V2FULL0, O_V2FULL1, O_D1FULL0, O_D1FULL1, O_D1EMPTY0, O_D1EMPTY1, O_D2FULL,
             O_D2EMPTY = O_D2FULL + 4, O_EPI = O_D2EMPTY + 4, O_SLOT0 };

__device__ __forceinline__ bool oz_failed(const int* err) { return *(const volatile int*)err != 0; }

// 32 TMEM lanes x N columns; the caller waits (tcgen05.wait::ld)
__device__ __forceinline__ void oz_tmem_ld(uint32_t taddr, float (&v)[2]) {
  uint32_t r[2];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
  v[0] = __uint_as_float(r[0]);
  v[1] = __uint_as_float(r[1]);
}
__device__ __forceinline__ void oz_tmem_ld(uint32_t taddr, float (&v)[4]) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;\n" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}

// group sums D_g (whole numbers) -> T 2^(-8 max(S-4, 0)), T = sum_g D_g 2^(8(S-1-g)):
// combined in 64-bit integers, then two FP64 additions (the integers are
// placed in the mantissa of 1.5 2^52 and 1.5 2^28)
template <int S>
__device__ __forceinline__ double oz_sum(const float (&d)[S]) {
  long long hi = (long long)__float2int_rn(d[3]);
  hi = mad_wide(__float2int_rn(d[2]), 1 << 8, hi);
  hi = mad_wide(__float2int_rn(d[1]), 1 << 16, hi);
  hi = mad_wide(__float2int_rn(d[0]), 1 << 24, hi);
  if constexpr (S == 4) {
    return __longlong_as_double(0x4338000000000000ll + hi) - 6755399441055744.0;
  } else {
    long long lo = (long long)__float2int_rn(d[6]);
    lo = mad_wide(__float2int_rn(d[5]), 1 << 8, lo);
    lo = mad_wide(__float2int_rn(d[4]), 1 << 16, lo);
    const double x = __longlong_as_double(0x4338000000000000ll + hi) - (6755399441055744.0 + 402653184.0);
    return x + __longlong_as_double(0x41B8000000000000ll + lo);
  }
}
// the same rounded to the vectors' type (FP32: without the FP64 pipe)
template <int S, typename T> __device__ __forceinline__ T oz_round(const float (&d)[S]) {
  if constexpr (std::is_same<T, double>::value) {
    return oz_sum<S>(d);
  } else {
    static_assert(S == 4, "FP32 results come from four digits");
    long long hi = (long long)__float2int_rn(d[3]);
    hi = mad_wide(__float2int_rn(d[2]), 1 << 8, hi);
    hi = mad_wide(__float2int_rn(d[1]), 1 << 16, hi);
    hi = mad_wide(__float2int_rn(d[0]), 1 << 24, hi);
    return __ll2float_rn(hi);
  }
}
// weight exponent of oz_sum's unit against scaled operands |v| < 1
template <int S> __host__ __device__ constexpr int oz_unit() { return -14 - 8 * (S - 1) + (S == 7 ? 24 : 0); }

// the same of NH columns of a TMEM accumulator region
template <int S, int NP, int NH, typename TR>
__device__ __forceinline__ void oz_combine(uint32_t taddr, TR (&t)[NH]) {
  float d[S][NH];
#pragma unroll
  for (int gI = 0; gI < S; ++gI) oz_tmem_ld(taddr + (uint32_t)(gI * NP), d[gI]);
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int j = 0; j < NH; ++j) {
    float x[S];
#pragma unroll
    for (int gI = 0; gI < S; ++gI) x[gI] = d[gI][j];
    t[j] = oz_round<S, TR>(x);
  }
}

// S digits, NP columns per pass, MS 128-value groups at most
template <int S, int NP, int MS, typename T, typename TA>
__global__ void __launch_bounds__(OZ_THREADS, 1)
    k_sigma_oz(OzGeom g, const OzItem* __restrict__ items, int nitems, int ngrp, OzShape sh, const uint16_t* __restrict__ dig, const int16_t* __restrict__ rexp,
               const int* __restrict__ ivexp, const T* __restrict__ diag, const T* __restrict__ V, int64_t ldv, int m, T* __restrict__ W,
               int64_t ldw, TA* __restrict__ W1, int64_t ld1, int* __restrict__ err) {
  constexpr int DW = oz_dw<S, NP>();
  constexpr int XR = oz_xrows<S, NP>();            // rows of the vector operands
  constexpr int PAD = oz_pad<NP>();
  constexpr int BOXB = XR * 128;
  constexpr int V2B = 2 * BOXB;
  constexpr int NH = NP / 4;                       // columns per epilogue thread
  constexpr int FB = 8 * S - 1;                    // fraction bits of the digits
  constexpr int TSH = oz_unit<S>();
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sX = base;                        // 2 nslot boxes [XR rows x 64 k]
  unsigned char* sV2 = base + sh.off_v2;           // nb x 2 boxes [XR rows x 64 tile rows]
  unsigned char* sRing = base + sh.off_ring;       // nr x 32 KB
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + sh.off_bar);
  uint64_t* slot_full = bars + O_SLOT0;
  uint64_t* slot_empty = slot_full + OZ_MAXNR;
  int* sXe = reinterpret_cast<int*>(slot_empty + OZ_MAXNR);    // [NP] exponents of X
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(sXe + NP);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int no = g.no, nv = g.nv, nvP = g.nvP;
  const int64_t n1 = g.n1;
  const int nunits = nitems * ngrp;

  if (tid == 0) {
    for (int i = 0; i < O_SLOT0 + 2 * OZ_MAXNR; ++i) {
      const bool epi = i == O_XFULL || i == O_V2FULL0 || i == O_V2FULL1 || i == O_D1EMPTY0 || i == O_D1EMPTY1 ||
                       (i >= O_D2EMPTY && i <= O_EPI);
      mbar_init(&bars[i], epi ? (uint32_t)OZ_EPI : 1u);
    }
  }
  if (warp == 0) tmem_alloc(tmem_holder, 512);
  // rows of the vector operands past S NP columns stay zero; so does, until a
  // full group overwrites it, the second box of a slot (a group of one box
  // leaves it as it is: its W1 lanes are not read)
  for (uint32_t o = tid; o < sh.off_bar / 16; o += OZ_THREADS) reinterpret_cast<uint4*>(base)[o] = make_uint4(0, 0, 0, 0);
  fence_proxy_async();
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tbase = *tmem_holder;
  const uint32_t tD2 = tbase + (uint32_t)(sh.nb * DW);         // + s DW

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      uint32_t use = 0;
      bool ok = true;
      for (int un = blockIdx.x; ok && un < nunits; un += gridDim.x) {
        const OzItem item = items[un / ngrp];
        const int nbox = ((item.holes & OZ_TWO ? 2 : 1) * nvP + OZ_BOX - 1) / OZ_BOX, nslot = (nbox + 1) / 2;
        const uint16_t* tp = dig + (int64_t)item.tile * (S * OZ_ROWS * OZ_BOX);
        for (int row0 = item.row0; ok && row0 < item.row1; row0 += OZ_ROWS) {
          for (int s = 0; ok && s < nslot; ++s) {
            const uint32_t bytes = 2 * s + 1 < nbox ? OZ_SLOT_BYTES : OZ_SLOT_BYTES / 2;
            for (int i = 0; i < S; ++i, ++use) {
              const uint32_t ri = use % sh.nr;
              ok = !oz_failed(err) && mbar_wait(&slot_empty[ri], ((use / sh.nr) & 1u) ^ 1u, err, 1);
              if (!ok) break;
              mbar_expect_tx(&slot_full[ri], bytes);
              bulk_load(sRing + (size_t)ri * OZ_SLOT_BYTES, tp, bytes, &slot_full[ri]);
              tp += bytes / 2;
            }
          }
        }
      }
      // no copy may still be writing shared memory when the CTA exits
      for (uint32_t k = 0; k < (uint32_t)sh.nr && k < use; ++k) {
        const uint32_t u = use - 1 - k;
        mbar_wait(&slot_full[u % sh.nr], (u / sh.nr) & 1u, err, 11);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA issuer
    // The whole warp walks the loops, so that descriptors and addresses stay
    // in uniform registers; one elected lane issues.  (One lane walking them
    // alone spent about 140 cycles an instruction and bound the pass.)
    constexpr uint64_t KMAJ = sdesc(0, 16, 1024, LAYOUT_SW128), MNMAJ = sdesc(0, OZ_SLOT_BYTES / 2, 1024, LAYOUT_SW128);
    const uint32_t sXa = smem_u32(sX), sVa = smem_u32(sV2), sRa = smem_u32(sRing);
    uint32_t ri = 0, rph = 0, tile = 0, nun = 0;
    uint32_t d2use[MS] = {};
    bool ok = true;
    for (int un = blockIdx.x; un < nunits && ok && !__any_sync(0xffffffffu, oz_failed(err)); un += gridDim.x, ++nun) {
      const OzItem item = items[un / ngrp];
      const int K = (item.holes & OZ_TWO ? 2 : 1) * nvP;
      const int nbox = (K + OZ_BOX - 1) / OZ_BOX, nslot = (nbox + 1) / 2;
      ok = mbar_wait_warp(&bars[O_XFULL], nun & 1u, err, 2);
      for (int row0 = item.row0; ok && row0 < item.row1; row0 += OZ_ROWS, ++tile) {
        const uint32_t b = sh.nb == 2 ? tile & 1u : 0u, ph = sh.nb == 2 ? (tile >> 1) & 1u : tile & 1u;
        ok = mbar_wait_warp(&bars[O_D1EMPTY0 + b], ph ^ 1u, err, 4);
        ok = ok && mbar_wait_warp(&bars[O_V2FULL0 + b], ph, err, 5);
        fence_after_sync();
        const uint32_t tD1 = tbase + b * DW;
        const uint64_t vdesc = KMAJ + ((sVa + b * V2B) >> 4);
        // the W1 sums run over OZ_FLUSH tiles of the item
        const int pos = ((row0 - item.row0) / OZ_ROWS) % OZ_FLUSH;
        const bool d2first = pos == 0, d2last = pos == OZ_FLUSH - 1 || row0 + OZ_ROWS >= item.row1;
#pragma unroll
        for (int s = 0; s < MS; ++s) {
          if (!ok || s >= nslot) break;
          if (d2first) {
            ok = mbar_wait_warp(&bars[O_D2EMPTY + s], (d2use[s] & 1u) ^ 1u, err, 3);
            ++d2use[s];
            fence_after_sync();
          }
          const uint64_t xdesc = KMAJ + ((sXa + 2 * s * BOXB) >> 4);
          const bool two = 2 * s + 1 < nbox;
#pragma unroll
          for (int i = 0; i < S; ++i) {
            ok = ok && mbar_wait_warp(&slot_full[ri], rph, err, 6);
            if (!ok) break;
            fence_after_sync();
            const uint32_t slot = sRa + ri * OZ_SLOT_BYTES;
            const uint32_t idK = idesc_bf16(OZ_ROWS, oz_n<S, NP>(i), 0, 0);
            const uint32_t idM = idesc_bf16(OZ_ROWS, oz_n<S, NP>(i), 1, 0);
            const uint32_t d1 = tD1 + (uint32_t)oz_col<NP>(i), d2 = tD2 + (uint32_t)(s * DW + oz_col<NP>(i));
            const uint64_t kd = KMAJ + (slot >> 4), md = MNMAJ + (slot >> 4);
            const uint64_t xd = xdesc + oz_brow<NP>(i) * 8, vd = vdesc + oz_brow<NP>(i) * 8;
            if (elect_one()) {
              // W2 tile: the slot's boxes as K-major A, X slices 0 .. S-1-i as B
              if (s == 0 && i == 0) mma_bf16_c<false>(d1, kd, xd, idK);
              else mma_bf16_c<true>(d1, kd, xd, idK);
#pragma unroll
              for (int ks = 1; ks < 4; ++ks) mma_bf16_c<true>(d1, kd + 2 * ks, xd + 2 * ks, idK);
              if (two) {
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                  mma_bf16_c<true>(d1, kd + OZ_SLOT_BYTES / 32 + 2 * ks, xd + BOXB / 16 + 2 * ks, idK);
              }
              // W1 part: the slot's 128 values of a as MN-major A, the tile's
              // 128 rows as K, V2 slices 0 .. S-1-i as B
              if (i == 0 && d2first) mma_bf16_c<false>(d2, md, vd, idM);
              else mma_bf16_c<true>(d2, md, vd, idM);
#pragma unroll
              for (int ks = 1; ks < 8; ++ks)
                mma_bf16_c<true>(d2, md + 128 * ks, vd + (ks >> 2) * (BOXB / 16) + 2 * (ks & 3), idM);
              mma_commit(&slot_empty[ri]);
              if (i == S - 1 && d2last) mma_commit(&bars[O_D2FULL + s]);
            }
            __syncwarp();
            if (++ri == (uint32_t)sh.nr) { ri = 0; rph ^= 1u; }
          }
        }
        if (elect_one()) mma_commit(&bars[O_D1FULL0 + b]);
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // thread = TMEM lane (tile row, or value index of a W1 group) and a
    // quarter of the columns
    const int ew = warp - 2;
    const int q = warp & 3;
    const int cbeg = (ew >> 2) * NH;
    const int r = 32 * q + lane;
    const uint32_t lane_off = (uint32_t)(32 * q) << 16;
    uint32_t tile = 0;
    uint32_t d2use[MS] = {};
    bool ok = true;
    int rx = 0;                 // exponent of the row of the tile being prepared
    T v2[NH];
    // V2 of a tile: this thread's row and columns
    auto load_v2 = [&](const OzItem& item, int row, int c0) {
      const bool valid = row < item.row1;
      const int64_t d = valid ? item.dbase + (int64_t)(row - item.row0) * item.dstr : 0;
      rx = valid ? (int)rexp[row - g.row0] : OZ_EMIN;
#pragma unroll
      for (int j = 0; j < NH; ++j) {
        const int c = c0 + cbeg + j;
        v2[j] = (valid && c < m) ? __ldg(V + (int64_t)c * ldv + n1 + d) : T(0);
      }
    };
    // all epilogue threads (an mbarrier, so that the wait is bounded)
    uint32_t nepi = 0;
    auto epi_sync = [&]() {
      mbar_arrive(&bars[O_EPI]);
      ok = mbar_wait_warp(&bars[O_EPI], nepi & 1u, err, 12) && ok;
      ++nepi;
    };
    int vexp[NH];               // exponents of the item's V2 columns
    auto store_v2 = [&](uint32_t buf) {
      unsigned char* bx = sV2 + buf * V2B + (r >> 6) * BOXB;
#pragma unroll
      for (int j = 0; j < NH; ++j) {
        const unsigned long long u =
            oz_fixed<S, T>(vexp[j] == OZ_NONFINITE ? T(0) : v2[j], FB - vexp[j] + rx);
#pragma unroll
        for (int i = 0; i < S; ++i)
          *reinterpret_cast<uint16_t*>(bx + sw128_off(PAD + i * NP + cbeg + j, r & 63)) = (uint16_t)(oz_digit<S>(u, i) >> 16);
      }
      fence_proxy_async();
      mbar_arrive(&bars[O_V2FULL0 + buf]);
    };
    for (int un = blockIdx.x; un < nunits && ok && !__any_sync(0xffffffffu, oz_failed(err)); un += gridDim.x) {
      const OzItem item = items[un / ngrp];
      const int c0 = (un % ngrp) * NP;
      const int K = (item.holes & OZ_TWO ? 2 : 1) * nvP;
      const int nbox = (K + OZ_BOX - 1) / OZ_BOX, nslot = (nbox + 1) / 2;
      const int kp = item.holes & 255, lp = (item.holes >> 8) & 255;
      load_v2(item, item.row0 + r, c0);
#pragma unroll
      for (int j = 0; j < NH; ++j)
        vexp[j] = c0 + cbeg + j < m ? __ldg(ivexp + (int64_t)(un / ngrp) * m + c0 + cbeg + j) : 0;
      // X of this item: the previous item's products have read the old one
      // (its last D1 was waited for).  One warp per column
#pragma unroll 1
      for (int c = ew; c < NP; c += OZ_EPI / 32) {
        T xv[4 * MS];
        int mx = OZ_EMIN;
#pragma unroll
        for (int u = 0; u < 4 * MS; ++u) {
          const int k = lane + 32 * u;
          const int seg = k >= nvP ? 1 : 0, a = k - seg * nvP;
          xv[u] = (c0 + c < m && k < K && a < nv) ? __ldg(V + (int64_t)(c0 + c) * ldv + (int64_t)a * no + (seg ? lp : kp)) : T(0);
        }
#pragma unroll
        for (int u = 0; u < 4 * MS; ++u) mx = max(mx, Parts<T>::exponent(xv[u]));
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) sXe[c] = mx;
#pragma unroll
        for (int u = 0; u < 4 * MS; ++u) {
          const int k = lane + 32 * u;
          if (k >= nbox * OZ_BOX) continue;
          const unsigned long long x = oz_fixed<S, T>(mx == OZ_NONFINITE ? T(0) : xv[u], FB - mx);
          unsigned char* bx = sX + (k >> 6) * BOXB;
#pragma unroll
          for (int i = 0; i < S; ++i)
            *reinterpret_cast<uint16_t*>(bx + sw128_off(PAD + i * NP + c, k & 63)) = (uint16_t)(oz_digit<S>(x, i) >> 16);
        }
      }
      fence_proxy_async();
      mbar_arrive(&bars[O_XFULL]);
      double acc[MS][NH];
#pragma unroll
      for (int s = 0; s < MS; ++s)
#pragma unroll
        for (int j = 0; j < NH; ++j) acc[s][j] = 0.0;
      epi_sync();               // sXe
      if (!ok) break;
      uint32_t buf = sh.nb == 2 ? tile & 1u : 0u;
      store_v2(buf);
      for (int row0 = item.row0; ok && row0 < item.row1; row0 += OZ_ROWS, ++tile) {
        buf = sh.nb == 2 ? tile & 1u : 0u;
        const uint32_t ph = sh.nb == 2 ? (tile >> 1) & 1u : tile & 1u;
        const bool has_next = row0 + OZ_ROWS < item.row1;
        const int rx_t = rx;
        const bool d2last = ((row0 - item.row0) / OZ_ROWS) % OZ_FLUSH == OZ_FLUSH - 1 || !has_next;
        if (has_next) load_v2(item, row0 + OZ_ROWS + r, c0);
        // W1 sums of one 128-value group
        auto drain_d2 = [&](int s, double (&ac)[NH]) {
          ok = ok && mbar_wait_warp(&bars[O_D2FULL + s], d2use[s] & 1u, err, 10);
          if (!ok) return;
          ++d2use[s];
          fence_after_sync();
          double t[NH];
          oz_combine<S, NP, NH, double>(tD2 + (uint32_t)(s * DW) + lane_off + (uint32_t)cbeg, t);
          fence_before_sync();
          mbar_arrive(&bars[O_D2EMPTY + s]);
#pragma unroll
          for (int j = 0; j < NH; ++j) ac[j] += t[j];
        };
#pragma unroll
        for (int s = 0; s + 1 < MS; ++s)
          if (d2last && s + 1 < nslot) drain_d2(s, acc[s]);
        // two buffers: the other one is free since the previous tile's end
        if (has_next && sh.nb == 2) store_v2(buf ^ 1u);
        ok = ok && mbar_wait_warp(&bars[O_D1FULL0 + buf], ph, err, 9);
        if (!ok) break;
        if (has_next && sh.nb == 1) store_v2(0);
        fence_after_sync();
        T t2[NH];
        oz_combine<S, NP, NH, T>(tbase + buf * DW + lane_off + (uint32_t)cbeg, t2);
        fence_before_sync();
        mbar_arrive(&bars[O_D1EMPTY0 + buf]);
        // the last group of the row (its sums end with the tile)
#pragma unroll
        for (int s = 0; s < MS; ++s)
          if (d2last && s + 1 == nslot) drain_d2(s, acc[s]);
        if (!ok) break;
        const int row = row0 + r;
        if (row < item.row1) {
          const int64_t d = item.dbase + (int64_t)(row - item.row0) * item.dstr;
          const T dg = diag[n1 + d];
          const int re = rx_t == 32767 ? OZ_NONFINITE : rx_t;
#pragma unroll
          for (int j = 0; j < NH; ++j) {
            const int c = c0 + cbeg + j;
            if (c >= m) continue;
            const T x = V[(int64_t)c * ldv + n1 + d];
            const T t = oz_scaled(t2[j], sXe[cbeg + j] + re + TSH);
            W[(int64_t)c * ldw + n1 + d] = dg * x + t;
          }
        }
      }
      if (!ok) break;
      // every thread is past its reads of sXe before the next item's X
      epi_sync();
#pragma unroll
      for (int s = 0; s < MS; ++s) {
        if (s >= nslot) continue;
        const int k = 128 * s + r;
        const int seg = k >= nvP ? 1 : 0, a = k - seg * nvP;
        if (k >= K || a >= nv) continue;
        const int64_t single = (int64_t)a * no + (seg ? lp : kp);
#pragma unroll
        for (int j = 0; j < NH; ++j) {
          const int c = c0 + cbeg + j;
          const double w = oz_scaled(acc[s][j], vexp[j] + TSH);
          if (c < m && !(w == 0.0)) atomicAdd(&W1[(int64_t)c * ld1 + single], (TA)w);
        }
      }
    }
  }
  // every role is done (or gave up): release TMEM
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  if (warp == 0) {
    tmem_dealloc(tbase, 512);
    tmem_relinquish();
  }
}

// ---------------------------------------------------------------------------
// Segments A and B: singles (a', k) and (b', k) of the classes with a' < b'.
//
// A run is the rows of one slab with equal a' (segment A; consecutive rows)
// or equal b' (segment B), coupled to the singles (f, k) of that fixed
// virtual f.  With R the run's rows x nocc segment values the products are
//   W2[r, c] += sum_k R[r, k] V[(f, k), c]
//   W1[(f, k), c] += sum_r R[r, k] V2[r, c]
// nocc is too short for a tcgen05 tile, so one warp takes a run and 16
// columns with mma.sync m16n8k16 on the same digits: 16 rows a step, staged
// by cp.async, their digits read by ldmatrix for W2 (K = k) and transposed
// for W1 (K = rows); the vectors' digits are made in registers.
// On the FP64 pipe the two segments took 34 of 50 ms (40 columns at
// nocc=16/nvirt=180).
// ---------------------------------------------------------------------------

// digits of the segments: [row - row0][segment A, B][slice][kw], kw = nocc
// rounded up to 16; one exponent per row over both segments
template <typename TV, int S>
__global__ void __launch_bounds__(256) k_oz_seg_values(GeomDev g, int64_t row0, int64_t row1, int kw,
                                                       const TV* __restrict__ Bt, uint16_t* __restrict__ out,
                                                       int16_t* __restrict__ sexp) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t row = row0 + ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5); row < row1; row += nw) {
    const int cls = row < g.start[1] ? 0 : row < g.start[2] ? 1 : row < g.start[3] ? 2 : row < g.start[4] ? 3 : 4;
    if (!(cls == 1 || cls >= 3)) continue;
    const TV* src = Bt + g.off[cls] + (row - g.start[cls]) * g.len[cls];
    uint16_t* o = out + (row - row0) * 2 * S * kw;
    int mx = OZ_VALUE_EMIN;
    for (int x = lane; x < 2 * kw; x += 32) {
      const int seg = x >= kw ? 1 : 0, k = x - seg * kw;
      if (k < g.no) mx = max(mx, Parts<TV>::exponent(src[seg * g.noP + k]));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) sexp[row - row0] = (int16_t)min(mx, 32767);
    for (int x = lane; x < 2 * kw; x += 32) {
      const int seg = x >= kw ? 1 : 0, k = x - seg * kw;
      const unsigned long long u = oz_fixed_value<S, TV>(k < g.no ? src[seg * g.noP + k] : TV(0), 8 * S - 1 - mx);
#pragma unroll
      for (int i = 0; i < S; ++i) o[(seg * S + i) * kw + k] = (uint16_t)(oz_digit<S>(u, i) >> 16);
    }
  }
}

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_seg(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int SEG_WARPS = 4;   // two a run
template <int S, int KT> __host__ __device__ constexpr int seg_pitch() { return S * KT * 32 + 16; }   // bytes of a staged row

// resident blocks the register budget is set for: 128 registers a thread where
// the slices of one k tile fit
template <int KT> __host__ __device__ constexpr int seg_blocks() { return KT == 1 ? 4 : 2; }

// exponent of a column over the four lanes that hold it
__device__ __forceinline__ int quad_max(int e) {
  e = max(e, __shfl_xor_sync(0xffffffffu, e, 1));
  return max(e, __shfl_xor_sync(0xffffffffu, e, 2));
}

// digits of 8 vector values as A fragments of m16n8k16: columns c = lane / 4
// and + 8, positions p = 2 (lane % 4), + 1, + 8, + 9; x[2 h + v] is position
// v of column half h (v = 0..3 in that order), sc[v] its power-of-two scale
template <int S, typename T>
__device__ __forceinline__ void seg_fragments(const T (&x)[2][4], const int (&sc)[4], const int (&ex)[2],
                                              uint32_t (&f)[S][4]) {
  unsigned long long u[2][4];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int v = 0; v < 4; ++v)
      u[h][v] = oz_fixed<S, T>(ex[h] == OZ_NONFINITE ? T(0) : x[h][v], 8 * S - 1 - ex[h] + sc[v]);
#pragma unroll
  for (int i = 0; i < S; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      f[i][h] = oz_pair(oz_digit<S>(u[h][0], i), oz_digit<S>(u[h][1], i));
      f[i][2 + h] = oz_pair(oz_digit<S>(u[h][2], i), oz_digit<S>(u[h][3], i));
    }
}

// SEGB: runs of equal b' (segment B), else of equal a' (segment A).  Two warps
// a run: the even one takes its W1 sums, the odd one its W2 rows, each with
// its own stage of the digits (the second read comes from L2).  One warp for
// both held 250 registers, eight warps an SM that spent 2.6 of their 5 stall
// cycles on fixed-latency results: 30 columns at nocc=13/nvirt=131 in 6.85 ms
// for the whole product, 5.82 with two warps.  Staging V2 and W2 of eight
// neighbouring runs through shared memory made segment B 7% faster and A 20%
// slower.
template <int S, int KT, bool SEGB, typename T, typename TA>
__global__ void __launch_bounds__(32 * SEG_WARPS, seg_blocks<KT>())
    k_oz_seg(OzGeom g, const OzSlab* __restrict__ slabs, int nslab, int ngrp, int item0,
             const uint16_t* __restrict__ dig, const int16_t* __restrict__ sexp, const int* __restrict__ vsexp, const T* __restrict__ V, int64_t ldv,
             int m, T* __restrict__ W, int64_t ldw, TA* __restrict__ W1, int64_t ld1) {
  constexpr int PITCH = seg_pitch<S, KT>(), NPIECE = 16 * S * KT * 2, KW = 16 * KT, TSH = oz_unit<S>();
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  const uint32_t sbase = smem_u32(smem + wid * 2 * 16 * PITCH);
  const int no = g.no, nv = g.nv;
  const int64_t n1 = g.n1;
  const int64_t nrun = (int64_t)nslab * ngrp * (nv - 1);
  // positions of this lane in a step of 16 rows (or singles)
  const int pos[4] = {2 * tig, 2 * tig + 1, 2 * tig + 8, 2 * tig + 9};
  for (int64_t run = blockIdx.x * (int64_t)(SEG_WARPS / 2) + (wid >> 1); run < nrun;
       run += (int64_t)gridDim.x * (SEG_WARPS / 2)) {
    const int fi = (int)(run % (nv - 1));
    const int64_t sg = run / (nv - 1);
    const int c0 = (int)(sg % ngrp) * 16;
    const OzSlab sl = slabs[sg / ngrp];
    const int f = SEGB ? fi + 1 : fi;
    const int nrow = SEGB ? f : nv - 1 - f;
    // slab-local pair of row t of the run; vector index of a pair
    auto pair_of = [&](int t) -> int64_t { return SEGB ? pair_index(t, f, nv) : pair_index(f, f + 1 + t, nv); };
    const int64_t dbase = n1 + sl.dbase;
    const int dstr = sl.dstr;
    const int64_t rloc = sl.row0 - g.row0;
    const int cc[2] = {c0 + gid, c0 + gid + 8};
    auto issue = [&](int t0, int b) {
      for (int p = lane; p < NPIECE; p += 32) {
        const int rr = p / (S * KT * 2), w = p - rr * (S * KT * 2);
        const bool ok = t0 + rr < nrow;
        const uint16_t* src = dig + ((rloc + (ok ? pair_of(t0 + rr) : 0)) * 2 + (SEGB ? 1 : 0)) * (S * KW) + 8 * w;
        const uint32_t dst = sbase + (uint32_t)((b * 16 + rr) * PITCH + 16 * w);
        const int n = ok ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n));
      }
      asm volatile("cp.async.commit_group;\n" ::);
    };
    __syncwarp();
    issue(0, 0);
    if (!(wid & 1)) {
      // ---- W1[(f, k), c] += sum_t R[t, k] V2[t, c]
      // column exponents of the slab's 2^er V2
      int ev[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        int e = cc[h] < m ? OZ_EMIN : 0;
        if (cc[h] < m)
          for (int i = 0; i < sl.nitem; ++i) e = max(e, __ldg(vsexp + (int64_t)(sl.item0 - item0 + i) * m + cc[h]));
        ev[h] = e;
      }
      float a1[2 * KT][S][4];
#pragma unroll
      for (int n = 0; n < 2 * KT; ++n)
#pragma unroll
        for (int i = 0; i < S; ++i) a1[n][i][0] = a1[n][i][1] = a1[n][i][2] = a1[n][i][3] = 0.f;
      for (int t0 = 0, b = 0; t0 < nrow; t0 += 16, b ^= 1) {
        __syncwarp();                                     // the other stage's readers are done
        if (t0 + 16 < nrow) issue(t0 + 16, b ^ 1);
        else asm volatile("cp.async.commit_group;\n" ::);
        T x[2][4];
        int er[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int t = t0 + pos[v];
          const bool ok = t < nrow;
          const int64_t pr = ok ? pair_of(t) : 0;
          er[v] = ok ? (int)sexp[rloc + pr] : OZ_EMIN;
#pragma unroll
          for (int h = 0; h < 2; ++h)
            x[h][v] = (ok && cc[h] < m) ? __ldg(V + (int64_t)cc[h] * ldv + dbase + pr * dstr) : T(0);
        }
        uint32_t vf[S][4];
        seg_fragments<S, T>(x, er, ev, vf);
        asm volatile("cp.async.wait_group 1;\n" ::);
        __syncwarp();
        // 16 x 16 digits of slice i, k group kt: row lane % 16, half lane / 16
        const uint32_t srow = sbase + (uint32_t)((b * 16 + (lane & 15)) * PITCH + (lane >> 4) * 16);
#pragma unroll
        for (int kt = 0; kt < KT; ++kt)
#pragma unroll
          for (int i = 0; i < S; ++i) {
            uint32_t q[4];
            ldsm_x4_t(q, srow + (i * KT + kt) * 32);      // (rows 0-7, 8-15) x k 0-7, then k 8-15
#pragma unroll
            for (int j = 0; j < S - i; ++j) {
              mma_seg(a1[2 * kt][i + j], vf[j], q[0], q[1]);
              mma_seg(a1[2 * kt + 1][i + j], vf[j], q[2], q[3]);
            }
          }
      }
#pragma unroll
      for (int n = 0; n < 2 * KT; ++n)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const int k = 8 * n + 2 * tig + v;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (k >= no || cc[h] >= m) continue;
            float dsum[S];
#pragma unroll
            for (int i = 0; i < S; ++i) dsum[i] = a1[n][i][2 * h + v];
            const double w = oz_scaled(oz_sum<S>(dsum), ev[h] + TSH);
            if (!(w == 0.0)) atomicAdd(&W1[(int64_t)cc[h] * ld1 + (int64_t)f * no + k], (TA)w);
          }
        }
    } else {
      // ---- W2[t, c] += sum_k R[t, k] V[(f, k), c]
      uint32_t xf[KT][S][4];
      int ex[2] = {OZ_EMIN, OZ_EMIN};
      {
        T x[KT][2][4];
#pragma unroll
        for (int kt = 0; kt < KT; ++kt)
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int k = 16 * kt + pos[v];
              x[kt][h][v] = (k < no && cc[h] < m) ? __ldg(V + (int64_t)cc[h] * ldv + (int64_t)f * no + k) : T(0);
              ex[h] = max(ex[h], Parts<T>::exponent(x[kt][h][v]));
            }
        ex[0] = quad_max(ex[0]);
        ex[1] = quad_max(ex[1]);
        const int sc0[4] = {0, 0, 0, 0};
#pragma unroll
        for (int kt = 0; kt < KT; ++kt) seg_fragments<S, T>(x[kt], sc0, ex, xf[kt]);
      }
      for (int t0 = 0, b = 0; t0 < nrow; t0 += 16, b ^= 1) {
        __syncwarp();
        if (t0 + 16 < nrow) issue(t0 + 16, b ^ 1);
        else asm volatile("cp.async.commit_group;\n" ::);
        // this step's W2 rows, ahead of their use
        int ee[4];
        T wv[2][4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int t = t0 + pos[v];
          const bool ok = t < nrow;
          const int64_t pr = ok ? pair_of(t) : 0;
          const int er = ok ? (int)sexp[rloc + pr] : OZ_EMIN;
          ee[v] = er == 32767 ? OZ_NONFINITE : er;
#pragma unroll
          for (int h = 0; h < 2; ++h)
            wv[h][v] = (ok && cc[h] < m) ? W[(int64_t)cc[h] * ldw + dbase + pr * dstr] : T(0);
        }
        asm volatile("cp.async.wait_group 1;\n" ::);
        __syncwarp();
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {                  // rows t0 + 8 hr ..
          float a2[S][4];
#pragma unroll
          for (int i = 0; i < S; ++i) a2[i][0] = a2[i][1] = a2[i][2] = a2[i][3] = 0.f;
          // two slices at a time: (slice i, k 0-7), (i, k 8-15), (i + 1, ..)
          const uint32_t srow2 = sbase + (uint32_t)((b * 16 + 8 * hr + (lane & 7)) * PITCH + ((lane >> 3) & 1) * 16);
#pragma unroll
          for (int kt = 0; kt < KT; ++kt)
#pragma unroll
            for (int i = 0; i < S; i += 2) {
              uint32_t q[4];
              const int i2 = i + 1 < S ? i + 1 : i;
              ldsm_x4(q, srow2 + (uint32_t)(((lane >> 4) ? i2 : i) * KT + kt) * 32);
#pragma unroll
              for (int j = 0; j < S - i; ++j) mma_seg(a2[i + j], xf[kt][j], q[0], q[1]);
              if (i + 1 < S) {
#pragma unroll
                for (int j = 0; j < S - i - 1; ++j) mma_seg(a2[i + 1 + j], xf[kt][j], q[2], q[3]);
              }
            }
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            const int t = t0 + 8 * hr + pos[v];
            if (t >= nrow) continue;
            const int64_t d = dbase + pair_of(t) * dstr;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (cc[h] >= m) continue;
              float dsum[S];
#pragma unroll
              for (int i = 0; i < S; ++i) dsum[i] = a2[i][2 * h + v];
              W[(int64_t)cc[h] * ldw + d] =
                  wv[h][2 * hr + v] + oz_scaled(oz_round<S, T>(dsum), ex[h] + ee[2 * hr + v] + TSH);
            }
          }
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
}

}  // namespace

// Digit store of the rows [row0, row1) of B^T and the work lists of the pass.
struct OzPlan {
  Ctx* ctx = nullptr;
  std::mutex mu;                      // held while a product is prepared and queued
  unsigned char* d_mem = nullptr;     // C|D digits, segment digits, their row exponents
  size_t mem_bytes = 0;
  bool refused = false;               // the digits did not fit when this matrix first asked
  uint16_t *dig = nullptr, *seg = nullptr;
  int16_t *rexp = nullptr, *sexp = nullptr;
  const void* values_for = nullptr;   // value store the digits were made of
  int S = 0;
  OzDst dst;
  OzGeom geom;
  unsigned char* d_lists = nullptr;   // work items, slabs, item exponents
  size_t list_bytes = 0;
  OzItem* items = nullptr;
  OzSlab* slabs = nullptr;
  int *vexp = nullptr, *vsexp = nullptr;
  std::vector<OzItem> h_items;        // host copies: all rows, in storage order
  std::vector<OzSlab> h_slabs;
  int item0 = 0, nitems = 0;          // those of the prepared rows
  int slab0 = 0, nslab = 0;
  int item_rows = 0, lists_m = 0;
};

// A context keeps the plan of a matrix that goes, with digits of up to this size,
// for its next one: their cudaMalloc (80 us for 9.5 MB) is most of what the first
// product of a small matrix takes beside a repeated one.  5/19, one column: 206 us
// with it, 129 without, 91 repeated (187 and 171 with the FP64 multiply-adds, which
// have no digits); 8/40: 378, 297, 186 (296, 275).
constexpr size_t OZ_SPARE_BYTES = (size_t)128 << 20;

// All plans of the process, for oz_reclaim.  Lock order: the registry, then one
// plan at a time; a thread that holds a plan's lock takes no other.
static std::mutex g_oz_mu;
static std::vector<OzPlan*> g_oz_plans;

std::unique_lock<std::mutex> oz_lock(Ctx* c, void*& handle) {
  OzPlan* p = reinterpret_cast<OzPlan*>(handle);
  if (!p && c->oz_spare) {
    p = reinterpret_cast<OzPlan*>(c->oz_spare);
    c->oz_spare = nullptr;
    handle = p;
  } else if (!p) {
    p = new OzPlan;
    p->ctx = c;
    const std::lock_guard<std::mutex> lock(g_oz_mu);
    g_oz_plans.push_back(p);
    handle = p;
  }
  return std::unique_lock<std::mutex>(p->mu);
}

// the digits (the plan's lock is held, and nothing queued reads them)
static void oz_drop_digits(OzPlan* p) {
  if (!p->d_mem) return;
  cudaFree(p->d_mem);
  p->ctx->oz_bytes -= (int64_t)p->mem_bytes;
  p->d_mem = nullptr;
  p->mem_bytes = 0;
  p->values_for = nullptr;
}

int64_t oz_reclaim(int device) {
  const std::lock_guard<std::mutex> registry(g_oz_mu);
  int64_t n = 0;
  for (OzPlan* p : g_oz_plans) {
    if (p->ctx->device != device) continue;
    const std::lock_guard<std::mutex> lock(p->mu);
    if (!p->d_mem) continue;
    n += (int64_t)p->mem_bytes;
    cudaStreamSynchronize(p->ctx->stream);   // its queued products
    oz_drop_digits(p);
  }
  return n;
}

void oz_free(Ctx* c, void*& handle, bool keep) {
  OzPlan* p = reinterpret_cast<OzPlan*>(handle);
  if (!p) return;
  if (keep && !c->oz_spare) {
    const std::lock_guard<std::mutex> lock(p->mu);
    if (p->d_mem && p->mem_bytes <= OZ_SPARE_BYTES) {
      dfree(c, p->d_lists);
      p->d_lists = nullptr;
      p->list_bytes = 0;
      p->item_rows = 0;
      p->refused = false;
      p->values_for = nullptr;
      c->oz_spare = p;
      handle = nullptr;
      return;
    }
  }
  {
    const std::lock_guard<std::mutex> registry(g_oz_mu);
    g_oz_plans.erase(std::find(g_oz_plans.begin(), g_oz_plans.end(), p));
  }
  oz_drop_digits(p);
  dfree(c, p->d_lists);
  delete p;
  handle = nullptr;
}

// no room for the work lists beside the digits
static int oz_give_up(Ctx* c, OzPlan* p) {
  ADC_CUDA(c, cudaStreamSynchronize(c->stream));
  oz_drop_digits(p);
  p->item_rows = 0;
  p->refused = true;
  return ADCGPU_OK;
}

// Room for the digits: a third of the device memory that is free now at most.
// The answer is kept for the matrix (until its digits are given back), so that
// its products do not change kernels with what else comes and goes on the device.
static int oz_room(Ctx* c, OzPlan* p, size_t bytes, bool* ok) {
  *ok = false;
  if (p->refused) return ADCGPU_OK;
  if (p->mem_bytes >= bytes) {
    *ok = true;
    return ADCGPU_OK;
  }
  // below 64 MB the question costs more than the answer is worth (40 us)
  if (bytes > (64u << 20)) {
    size_t free_b = 0, total_b = 0;
    ADC_CUDA(c, cudaMemGetInfo(&free_b, &total_b));
    if (bytes > (free_b + p->mem_bytes) / 3) {
      p->refused = true;
      return ADCGPU_OK;
    }
  }
  oz_drop_digits(p);
  const cudaError_t e = cudaMalloc((void**)&p->d_mem, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    p->d_mem = nullptr;
    p->refused = true;
    return ADCGPU_OK;
  }
  ADC_CUDA(c, e);
  p->mem_bytes = bytes;
  c->oz_bytes += (int64_t)bytes;
  *ok = true;
  return ADCGPU_OK;
}

void oz_invalidate(void* handle) {
  if (OzPlan* p = reinterpret_cast<OzPlan*>(handle)) p->values_for = nullptr;
}

// C|D rows of up to 512 values (nvirt <= 256), segments of up to 32: every
// system the library takes
bool oz_geometry_ok(const Geometry& G) { return G.no <= 32 && G.nv >= 2 && 2 * G.nvP <= 512; }

// Column counts from which the sliced pass is the faster one.  It reads 14 (8)
// bytes a value instead of 8 (4), pads segments A and B to 16 or 32 holes and
// computes 8 or 16 columns whatever m is; the per-warp passes below 16 columns
// take 4, 2 and 1 FP32 or 2 and 1 FP64 columns at a time.  Microseconds, per-warp
// / sliced, at nocc/nvirt:
//   FP64     10/110 m=1 1494/915; 5/19 m=1 166/89; 20/40 m=1 954/1150, m=2
//            1773/1164; 32/32 m=1 1472/2049; 18/90 m=1 3406/3324; 3/6 m=1 77/86, m=2 102/87
//   FP32     10/110 m=1 353/619, m=2 495/635, m=3 810/658, m=4 785/673; 8/40 m=2
//            110/145, m=3 171/152; 5/130 m=3 394/379, m=4 326/388; 18/90 m=4
//            1713/2188, m=8 3378/2246; 32/32 m=5 1113/1409, m=8 1531/1414; 2/6 m=4 61/87
//   direct   (digits made in every product) 10/110 m=1 3805/4501, m=2 5357/4539;
//            18/90 m=1 8015/10246, m=2 11223/10286; 5/19 m=1 737/1367, m=4 2292/1405
bool oz_faster(const Ctx* c, bool f64, int m) {
  const Geometry& G = c->geom;
  if (c->oz_always) return true;
  if (f64) return m > (c->direct || G.no > 16 ? 1 : 0) && m * G.nv >= 8;
  // (tiny systems: the fixed time of the launches decides)
  const int passes = m < 16 ? m / 4 + (m >> 1 & 1) + (m & 1) : (m + 15) / 16;
  return m >= (G.no > 16 ? 6 : 3) && passes * G.nv > 12;
}

// The same for the CVS matrix against its compressed rows: an entry costs the row
// kernel 11.5 ps a column, a row the sliced pass 0.85 ns more, and its launches
// 25 us more.  (8/40, 1 core orbital: 4 columns 61/80 us, 8 100/89; 9/107: one
// column 225/167; 14/60, 3 core orbitals: one column 158/200, two 239/201; 5/19,
// 3: 32 columns 92/107.)
bool oz_faster_cvs(const Ctx* c, int m) {
  return c->oz_always || c->cvs_nnz * m - 74 * (c->cvs_N - c->cvs_n1) >= 2200000;
}

namespace {

// rows of a typical range of the direct path: the digits of a range take about
// as many bytes as the FP64 values of a chunk, three times those of its rows
int64_t direct_range_rows(const Ctx* c) {
  int64_t rows = 1;
  for (const DirectChunk& d : c->dchunks) rows = std::max(rows, (d.row1 - d.row0) / 3);
  return rows;
}

size_t oz_digit_bytes(const Geometry& G, int64_t row0, int64_t row1, int S, OzDst* dst) {
  int64_t n = 0, tiles = 0;
  for (int cls = 0; cls < 5; ++cls) {
    const int64_t a = std::max(row0, G.start[cls]), b = std::min(row1, G.start[cls + 1]), sl = G.slab_len(cls);
    dst->base[cls] = n;
    dst->r0[cls] = a;
    dst->slab[cls] = sl;
    dst->tps[cls] = (int)((sl + OZ_ROWS - 1) / OZ_ROWS);
    dst->nbox[cls] = (int)(((cls >= 2 ? 2 : 1) * G.nvP + OZ_BOX - 1) / OZ_BOX);
    dst->tiles[cls] = tiles;
    const int64_t nt = a < b ? (b - a) / sl * dst->tps[cls] : 0;
    tiles += nt;
    n += nt * S * dst->nbox[cls] * OZ_ROWS * OZ_BOX;
  }
  dst->tiles[5] = tiles;
  dst->row0 = row0;
  dst->row1 = row1;
  return (size_t)n * sizeof(uint16_t);
}

size_t align256(size_t x) { return (x + 255) / 256 * 256; }

struct OzBytes { size_t dig, seg, exp, all; };
OzBytes oz_bytes(const Geometry& G, int64_t row0, int64_t row1, int S, OzDst* dst) {
  OzBytes b;
  const int kw = (G.no + 15) / 16 * 16;
  const size_t nrows = (size_t)(row1 - row0);
  b.dig = align256(oz_digit_bytes(G, row0, row1, S, dst));
  b.seg = align256(nrows * 2 * S * kw * sizeof(uint16_t));
  b.exp = align256(nrows * sizeof(int16_t));
  b.all = b.dig + b.seg + 2 * b.exp;
  return b;
}

}  // namespace

// The rows [row0, row1) as ranges of whole slabs whose digits are prepared
// and used together: one range for a stored matrix; on the direct path, whose
// point is a small footprint, ranges whose digits take no more than the chunk
// buffer (never less than one slab).  *reserve: the most that any range of the
// matrix takes.
std::vector<std::pair<int64_t, int64_t>> oz_ranges(const Ctx* c, int64_t row0, int64_t row1, int64_t* reserve) {
  const Geometry& G = c->geom;
  std::vector<std::pair<int64_t, int64_t>> out;
  *reserve = 0;
  if (!c->direct) {
    out.emplace_back(row0, row1);
    return out;
  }
  const int64_t budget = direct_budget(G) * (int64_t)sizeof(double);
  *reserve = budget;   // (the direct path computes in FP64: seven digits)
  for (int cls = 0; cls < 5; ++cls) {
    OzDst d;
    if (G.start[cls] < G.start[cls + 1])
      *reserve = std::max<int64_t>(*reserve, oz_bytes(G, G.start[cls], G.start[cls] + G.slab_len(cls), 7, &d).all);
  }
  int64_t used = 0;
  for (int cls = 0; cls < 5; ++cls) {
    const int64_t a = std::max(row0, G.start[cls]), b = std::min(row1, G.start[cls + 1]), sl = G.slab_len(cls);
    for (int64_t s0 = a; s0 < b; s0 += sl) {
      OzDst d;
      const int64_t n = (int64_t)oz_bytes(G, s0, s0 + sl, 7, &d).all;
      if (out.empty() || used + n > budget) {
        out.emplace_back(s0, s0);
        used = 0;
      }
      out.back().second = s0 + sl;
      used += n;
    }
  }
  return out;
}

namespace {

// an item's vector operand in tiles (about a third) and its last drains
constexpr double OZ_ITEM_OVERHEAD = 0.5;

// the work items of one slab, in equal pieces of whole tiles
void oz_add_slab(OzPlan* p, int64_t s0, int64_t len, int item_rows, int holes, bool pairs, int64_t dbase, int dstr) {
  const int64_t npc = (len + item_rows - 1) / item_rows;
  const int64_t per = ((len + npc - 1) / npc + OZ_ROWS - 1) / OZ_ROWS * OZ_ROWS;
  const int i0 = (int)p->h_items.size();
  for (int64_t x = 0; x < len; x += per)
    p->h_items.push_back(OzItem{(int)(s0 + x), (int)(s0 + std::min(x + per, len)), -1,
                                holes | (pairs ? OZ_PAIRS : 0), (int)(dbase + x * dstr), dstr, 0, 0});
  if (pairs)
    p->h_slabs.push_back(OzSlab{(int)s0, (int)dbase, dstr, i0, (int)p->h_items.size() - i0, 0, 0, 0});
}

int oz_upload_lists(Ctx* c, OzPlan* p, int item_rows, int m) {
  const size_t ni = p->h_items.size(), ns = p->h_slabs.size();
  const size_t ib = align256(sizeof(OzItem) * ni), lb = ib + align256(sizeof(OzSlab) * ns);
  const size_t need = lb + 2 * sizeof(int) * ni * m;
  if (p->list_bytes < need) {
    dfree(c, p->d_lists);
    p->d_lists = nullptr;
    p->list_bytes = 0;
    ST(dmalloc(c, (void**)&p->d_lists, need, false));   // (the plan is locked)
    p->list_bytes = need;
  }
  p->items = reinterpret_cast<OzItem*>(p->d_lists);
  p->slabs = reinterpret_cast<OzSlab*>(p->d_lists + ib);
  p->vexp = reinterpret_cast<int*>(p->d_lists + lb);
  p->vsexp = p->vexp + ni * m;
  std::vector<unsigned char> all(lb);
  std::copy_n(reinterpret_cast<const unsigned char*>(p->h_items.data()), sizeof(OzItem) * ni, all.data());
  std::copy_n(reinterpret_cast<const unsigned char*>(p->h_slabs.data()), sizeof(OzSlab) * ns, all.data() + ib);
  // pageable source: staged before the call returns, no need to wait
  ADC_CUDA(c, cudaMemcpyAsync(p->items, all.data(), lb, cudaMemcpyHostToDevice, c->stream));
  p->item_rows = item_rows;
  p->lists_m = m;
  return ADCGPU_OK;
}

}  // namespace

// Makes the digits of the rows [row0, row1) (kept until the values change;
// the direct path's chunk buffer is rewritten for every chunk) and the work
// lists of an m-column product.  reserve: bytes the digits of any range of
// this matrix may take.  *usable stays false, and the CUDA-core tile takes the
// product, for shapes the pass does not take and when there is no room for the
// digits.  The plan is locked (oz_lock).
int oz_prepare(Ctx* c, void*& handle, const void* values, bool f64, int64_t row0, int64_t row1, int64_t reserve, int m,
               bool* usable) {
  *usable = false;
  const Geometry& G = c->geom;
  if (!oz_geometry_ok(G)) return ADCGPU_OK;
  const int S = f64 ? 7 : 4;
  OzPlan* p = reinterpret_cast<OzPlan*>(handle);
  OzDst dst;
  const int kw = (G.no + 15) / 16 * 16;
  const OzBytes need = oz_bytes(G, row0, row1, S, &dst);
  bool room = false;
  ST(oz_room(c, p, std::max(need.all, (size_t)reserve), &room));
  if (!room) return ADCGPU_OK;
  if (!(p->values_for && p->values_for == values && p->S == S && p->dst.row0 == row0 && p->dst.row1 == row1)) {
    p->dst = dst;
    p->S = S;
    p->dig = reinterpret_cast<uint16_t*>(p->d_mem);
    p->seg = reinterpret_cast<uint16_t*>(p->d_mem + need.dig);
    p->rexp = reinterpret_cast<int16_t*>(p->d_mem + need.dig + need.seg);
    p->sexp = reinterpret_cast<int16_t*>(p->d_mem + need.dig + need.seg + need.exp);
    const GeomDev g = to_dev(G);
    const int grid = (int)std::min<int64_t>(dst.tiles[5] * OZ_ROWS / 8, (int64_t)c->nsm * 8);
    const int grid2 = (int)std::min<int64_t>((row1 - row0 + 7) / 8, (int64_t)c->nsm * 8);
    auto make = [&](auto* v, auto s) {
      using TV = typename std::remove_const<typename std::remove_pointer<decltype(v)>::type>::type;
      constexpr bool F64 = decltype(s)::value == 7;
      if (F64 && 2 * G.nvP > 256) k_oz_values<TV, decltype(s)::value, F64><<<grid, 256, 0, c->stream>>>(g, dst, v, p->dig, p->rexp);
      else k_oz_values<TV, decltype(s)::value, false><<<grid, 256, 0, c->stream>>>(g, dst, v, p->dig, p->rexp);
      ADC_COUNT_LAUNCH();
      k_oz_seg_values<TV, decltype(s)::value><<<grid2, 256, 0, c->stream>>>(g, row0, row1, kw, v, p->seg, p->sexp);
      ADC_COUNT_LAUNCH();
    };
    if (f64) make((const double*)values, std::integral_constant<int, 7>());
    else make((const float*)values, std::integral_constant<int, 4>());
    ADC_CUDA(c, cudaGetLastError());
    p->values_for = c->direct ? nullptr : values;
  }
  // an item's place in the digit store of the prepared rows
  auto set_tile = [&](OzItem& it) {
    int cls = 0;
    while (cls < 4 && it.row0 >= G.start[cls + 1]) ++cls;
    const int64_t rc = it.row0 - dst.r0[cls], slab = rc / dst.slab[cls];
    it.tile = (int)(dst.base[cls] / ((int64_t)S * OZ_ROWS * OZ_BOX) +
                    (slab * dst.tps[cls] + (rc - slab * dst.slab[cls]) / OZ_ROWS) * dst.nbox[cls]);
  };
  // slabs of pairs: classes 1, 4I and 4II (of the whole matrix, or as many as
  // a typical range of the direct path holds)
  const int64_t nslab = c->direct ? std::max<int64_t>(1, direct_range_rows(c) / std::max<int64_t>(1, G.npair_v))
                                  : G.no + 2 * G.npair_o;
  const int item_rows = item_rows_for(c, nslab, G.npair_v, (m + 15) / 16, OZ_ITEM_OVERHEAD);
  if (p->item_rows != item_rows || p->lists_m < m) {
    p->h_items.clear();
    p->h_slabs.clear();
    for (int cls = 0; cls < 5; ++cls) {
      const int64_t sl = G.slab_len(cls);
      for (int64_t s0 = G.start[cls], k = 0; s0 < G.start[cls + 1]; s0 += sl, ++k) {
        int kp = (int)k, lp = (int)k;
        if (cls >= 2) pair_decode(k, G.no, kp, lp);
        // class 2 (stored hole outer) is hole inner in the vectors
        oz_add_slab(p, s0, sl, item_rows, kp | lp << 8 | (cls >= 2 ? OZ_TWO : 0), cls == 1 || cls >= 3,
                    cls == 1 ? G.start[1] + k : s0, cls == 1 ? G.no : 1);
      }
    }
    if (!c->direct)
      for (OzItem& it : p->h_items) set_tile(it);
    const int st = oz_upload_lists(c, p, item_rows, m);
    if (st == ADCGPU_OUT_OF_MEMORY) return oz_give_up(c, p);
    ST(st);
  }
  // the prepared rows' items
  auto first = [](const auto& v, int64_t row) {
    return (int)(std::lower_bound(v.begin(), v.end(), row, [](const auto& a, int64_t r) { return a.row0 < r; }) - v.begin());
  };
  p->item0 = first(p->h_items, row0);
  p->nitems = first(p->h_items, row1) - p->item0;
  p->slab0 = first(p->h_slabs, row0);
  p->nslab = first(p->h_slabs, row1) - p->slab0;
  // a range of the direct path: its tiles, counted from the range's first
  // (the same in every product)
  if (c->direct && p->nitems && p->h_items[p->item0].tile < 0) {
    for (int i = p->item0; i < p->item0 + p->nitems; ++i) set_tile(p->h_items[i]);
    ADC_CUDA(c, h2d(c, p->items + p->item0, p->h_items.data() + p->item0, sizeof(OzItem) * (size_t)p->nitems));
  }
  p->geom = OzGeom{G.no, G.nv, G.nvP, G.n1, row0};
  *usable = true;
  return ADCGPU_OK;
}

// Digits and work lists of the CVS matrix's pair rows (spins I and II); the
// rows with a' = b' stay with the compressed-row kernel.
int oz_prepare_cvs(Ctx* c, void*& handle, int m, bool* usable) {   // (the plan is locked)
  *usable = false;
  const Geometry& G = c->geom;
  constexpr int S = 7;
  const int nc = (int)(c->cvs_n1 / G.nv), kw = 16 * ((nc + 15) / 16);
  std::vector<char> core(G.no, 0);
  for (int k = 0; k < nc; ++k) core[c->cvs_kpq[7 * (1 + k) + 2] - 1] = 1;   // holes of the first virtual's singles
  std::vector<int> index(G.no, -1), hole;                                   // hole pairs with one core orbital
  for (int i = 0, n = 0; i < G.no; ++i) if (core[i]) index[i] = n++;
  for (int i = 0; i < G.no; ++i)
    for (int j = i + 1; j < G.no; ++j)
      if (core[i] + core[j] == 1) hole.push_back(core[i] ? index[i] : index[j]);
  const int npp = (int)hole.size();
  const int64_t npair = G.npair_v, nrows = 2 * npp * npair, c3 = (int64_t)npp * G.nv;
  const int nbox = (G.nvP + OZ_BOX - 1) / OZ_BOX;
  const int64_t tps = (npair + OZ_ROWS - 1) / OZ_ROWS;
  if (nrows == 0 || c->cvs_N != c->cvs_n1 + c3 + nrows) return ADCGPU_OK;
  OzPlan* p = reinterpret_cast<OzPlan*>(handle);
  const size_t dig_b = align256(sizeof(uint16_t) * (size_t)(2 * npp * tps) * S * nbox * OZ_ROWS * OZ_BOX);
  const size_t seg_b = align256(sizeof(uint16_t) * (size_t)nrows * 2 * S * kw), exp_b = align256(sizeof(int16_t) * (size_t)nrows);
  bool room = false;
  ST(oz_room(c, p, dig_b + seg_b + 2 * exp_b, &room));
  if (!room) return ADCGPU_OK;
  p->geom = OzGeom{nc, G.nv, G.nvP, c->cvs_n1, 0};
  if (p->values_for != c->d_cval) {
    p->S = S;
    p->dig = reinterpret_cast<uint16_t*>(p->d_mem);
    p->seg = reinterpret_cast<uint16_t*>(p->d_mem + dig_b);
    p->rexp = reinterpret_cast<int16_t*>(p->d_mem + dig_b + seg_b);
    p->sexp = reinterpret_cast<int16_t*>(p->d_mem + dig_b + seg_b + exp_b);
    const int grid = (int)std::min<int64_t>(2 * npp * tps * OZ_ROWS / 4, (int64_t)c->nsm * 16);
    k_oz_cvs_values<S><<<grid, 128, sizeof(double) * 4 * (size_t)(G.nvP + 2 * kw), c->stream>>>(
        p->geom, npp, c3, c->d_crow, c->d_ccol, c->d_cval, kw, p->dig, p->seg, p->rexp, p->sexp);
    ADC_COUNT_LAUNCH();
    ADC_CUDA(c, cudaGetLastError());
    p->values_for = c->d_cval;
  }
  const int item_rows = item_rows_for(c, 2 * npp, npair, (m + 15) / 16, OZ_ITEM_OVERHEAD);
  if (p->item_rows != item_rows || p->lists_m < m) {
    p->h_items.clear();
    p->h_slabs.clear();
    for (int s = 0; s < 2 * npp; ++s) {
      const int first = (int)p->h_items.size();
      oz_add_slab(p, s * npair, npair, item_rows, hole[s % npp], true, c3 + s * npair, 1);
      for (int i = first; i < (int)p->h_items.size(); ++i)
        p->h_items[i].tile = (int)((s * tps + (p->h_items[i].row0 - s * npair) / OZ_ROWS) * nbox);
    }
    const int st = oz_upload_lists(c, p, item_rows, m);
    if (st == ADCGPU_OUT_OF_MEMORY) return oz_give_up(c, p);
    ST(st);
  }
  p->item0 = p->slab0 = 0;
  p->nitems = (int)p->h_items.size();
  p->nslab = (int)p->h_slabs.size();
  *usable = true;
  return ADCGPU_OK;
}

namespace {

// shared memory of one launch over rows of up to 'values' C|D values; nb = 2 where TMEM and shared memory hold two
// D1 / V2 buffers beside at least three ring slots; false when even one
// buffer does not fit
template <int S, int NP>
bool oz_shape(int values, int smax, OzShape* sh, size_t* bytes) {
  constexpr int DW = oz_dw<S, NP>(), BOXB = oz_xrows<S, NP>() * 128, V2B = 2 * BOXB;
  sh->nslot = (values + 127) / 128;
  const size_t tail = (size_t)(O_SLOT0 + 2 * OZ_MAXNR) * 8 + (size_t)NP * 4 + 16;
  for (sh->nb = 2; sh->nb >= 1; --sh->nb) {
    if ((sh->nb + sh->nslot) * DW > 512) continue;
    sh->off_v2 = (uint32_t)(2 * sh->nslot) * BOXB;
    sh->off_v2 = (sh->off_v2 + 1023) / 1024 * 1024;
    sh->off_ring = sh->off_v2 + (uint32_t)sh->nb * V2B;
    const int64_t room = (int64_t)smax - 1024 - (int64_t)tail - sh->off_ring;
    sh->nr = (int)std::min<int64_t>(OZ_MAXNR, room / OZ_SLOT_BYTES);
    if (sh->nr < (sh->nb == 2 ? 3 : 2)) continue;
    sh->off_bar = sh->off_ring + (uint32_t)sh->nr * OZ_SLOT_BYTES;
    *bytes = 1024 + sh->off_bar + tail;
    return true;
  }
  return false;
}

template <int S, int NP, int MS, typename T, typename TA>
int oz_go(Ctx* c, OzPlan* p, int smax, const OzShape& sh, size_t smem, const T* diag, const T* V, int64_t ldv, int m,
          T* W, int64_t ldw, TA* W1, int64_t ld1) {
  auto kern = k_sigma_oz<S, NP, MS, T, TA>;
  ADC_CUDA(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smax));
  const int ngrp = (m + NP - 1) / NP;
  const int grid = std::max(1, std::min(p->nitems * ngrp, c->nsm));
  k_oz_vexp<T><<<dim3(p->nitems, (m + 3) / 4), 256, 0, c->stream>>>(p->geom, p->items + p->item0, p->rexp, p->sexp, V,
                                                                    ldv, m, p->vexp, p->vsexp);
  ADC_COUNT_LAUNCH();
  kern<<<grid, OZ_THREADS, smem, c->stream>>>(p->geom, p->items + p->item0, p->nitems, ngrp, sh, p->dig, p->rexp,
                                              p->vexp, diag, V, ldv, m, W, ldw, W1, ld1, c->d_word);
  ADC_COUNT_LAUNCH();
  ADC_CUDA(c, cudaGetLastError());
  return ADCGPU_OK;
}

// segments A and B of m columns: W2 rows and W1 sums are added to
template <int S, int KT, bool SEGB, typename T, typename TA>
int oz_seg_go(Ctx* c, OzPlan* p, const T* V, int64_t ldv, int m, T* W, int64_t ldw, TA* W1, int64_t ld1) {
  auto kern = k_oz_seg<S, KT, SEGB, T, TA>;
  const size_t smem = (size_t)SEG_WARPS * 2 * 16 * seg_pitch<S, KT>();
  ADC_CUDA(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int ngrp = (m + 15) / 16;
  const int64_t nblk = ((int64_t)p->nslab * ngrp * (p->geom.nv - 1) + SEG_WARPS / 2 - 1) / (SEG_WARPS / 2);
  const int grid = (int)std::min<int64_t>(nblk, (int64_t)c->nsm * 16);
  kern<<<grid, 32 * SEG_WARPS, smem, c->stream>>>(p->geom, p->slabs + p->slab0, p->nslab, ngrp, p->item0, p->seg, p->sexp,
                                                  p->vsexp, V, ldv, m, W, ldw, W1, ld1);
  ADC_COUNT_LAUNCH();
  ADC_CUDA(c, cudaGetLastError());
  return ADCGPU_OK;
}

template <int S, typename T, typename TA>
int oz_seg(Ctx* c, OzPlan* p, const T* V, int64_t ldv, int m, T* W, int64_t ldw, TA* W1, int64_t ld1) {
  if (p->nslab == 0) return ADCGPU_OK;
  if (p->geom.no <= 16) {
    ST((oz_seg_go<S, 1, false>(c, p, V, ldv, m, W, ldw, W1, ld1)));
    return oz_seg_go<S, 1, true>(c, p, V, ldv, m, W, ldw, W1, ld1);
  }
  ST((oz_seg_go<S, 2, false>(c, p, V, ldv, m, W, ldw, W1, ld1)));
  return oz_seg_go<S, 2, true>(c, p, V, ldv, m, W, ldw, W1, ld1);
}

}  // namespace

// The coupling products of m columns over the prepared rows, segment A of
// the classes with a' = b' excepted: W2 rows are stored with the diagonal
// term, W1 sums are added.
int oz_launch(Ctx* c, void* handle, const double* diag, const double* V, int64_t ldv, int m, double* W, int64_t ldw,
              double* W1, int64_t ld1) {
  OzPlan* p = reinterpret_cast<OzPlan*>(handle);
  const int smax = smem_optin_max(c), values = (c->cvs ? 1 : 2) * p->geom.nvP;   // of the longest C|D row
  OzShape sh;
  size_t smem = 0;
  // 16 columns per pass where their accumulators fit (rows of up to 384
  // values); the column groups of an item run side by side, so the digits
  // come from L2 for all but one of them
  if (m > 8 && oz_shape<7, 16>(values, smax, &sh, &smem))
    ST((oz_go<7, 16, 3>(c, p, smax, sh, smem, diag, V, ldv, m, W, ldw, W1, ld1)));
  else if (oz_shape<7, 8>(values, smax, &sh, &smem))
    ST((oz_go<7, 8, 4>(c, p, smax, sh, smem, diag, V, ldv, m, W, ldw, W1, ld1)));
  else
    return set_err(c, ADCGPU_UNSUPPORTED, "sliced sigma pass: shape");
  return oz_seg<7>(c, p, V, ldv, m, W, ldw, W1, ld1);
}

// FP32 values and vectors (four digits), FP64 W1 accumulators
int oz_launch(Ctx* c, void* handle, const float* diag, const float* V, int64_t ldv, int m, float* W, int64_t ldw,
              double* W1, int64_t ld1) {
  OzPlan* p = reinterpret_cast<OzPlan*>(handle);
  const int smax = smem_optin_max(c), values = (c->cvs ? 1 : 2) * p->geom.nvP;   // of the longest C|D row
  OzShape sh;
  size_t smem = 0;
  if (!oz_shape<4, 16>(values, smax, &sh, &smem)) return set_err(c, ADCGPU_UNSUPPORTED, "sliced sigma pass: shape");
  ST((oz_go<4, 16, 4>(c, p, smax, sh, smem, diag, V, ldv, m, W, ldw, W1, ld1)));
  return oz_seg<4>(c, p, V, ldv, m, W, ldw, W1, ld1);
}

int sigma_queue_status(Ctx* c) {
  ADC_CUDA(c, cudaMemcpyAsync(c->h_word, c->d_word, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  ADC_CUDA(c, cudaEventRecord(c->word_ev, c->stream));
  c->word_pending = true;
  return ADCGPU_OK;
}

int sigma_status_so_far(Ctx* c) {
  if (!c->word_pending) return ADCGPU_OK;
  const cudaError_t e = cudaEventQuery(c->word_ev);
  if (e == cudaErrorNotReady) return ADCGPU_OK;
  ADC_CUDA(c, e);
  return *c->h_word ? sigma_status(c) : ADCGPU_OK;
}

int sigma_status(Ctx* c) {
  if (!c->word_pending) return ADCGPU_OK;
  ADC_CUDA(c, cudaStreamSynchronize(c->stream));
  c->word_pending = false;
  if (!*c->h_word) return ADCGPU_OK;
  const int code = *c->h_word;
  ADC_CUDA(c, cudaMemsetAsync(c->d_word, 0, sizeof(int), c->stream));
  return set_err(c, ADCGPU_DEVICE_TIMEOUT,
                 "tensor-core sigma pass: a pipeline wait timed out (stage " + std::to_string(code) + ")");
}

}  // namespace adcgpu
