// FP64-accurate GEMM on the 5th-generation tensor cores by exact digit
// slicing (the error-free splitting of Ozaki, Ogita, Oishi and Rump, 2012,
// with integer digits), for the FP64 contractions of the RI pipeline: the
// two transform_ri products (src/POSTHF/ri.cc:147-172) and the metric
// application B = L^-1 (P|ia) (the calculate_ri product, ri.cc:102-103).
//
// Slicing.  Per pass of 512 of K, row r of an operand is scaled by 2^-e_r (e_r:
// the binary exponent of its largest element there, so every scaled value lies
// in (-1, 1)) and written as eight balanced base-128 digits,
//   x / 2^e_r = sum_{s=0..7} d_s 2^(-7 (s+1)) + rho,  |d_0| <= 128,
//   |d_s| <= 64 (s >= 1),  |rho| <= 2^-57,
// computed with integer operations on the FP64 bit pattern (no FP64
// arithmetic: GB300 runs FP64 at 1/64 of the FP32 rate).  Digits are small
// integers, exact in BF16.
//
// Products.  C(m, n) = 2^(e_m + f_n) sum_L 2^(-7 (L+2)) acc_L(m, n) with the
// level sums acc_L = sum_{s+t=L} sum_k d_s(A)[m][k] d_t(B)[n][k], L = 0..7
// (36 digit products; the levels L >= 8 fall below 2^-56 of the row and
// column scales).  With K <= 512 per pass every level L <= 5 stays below 2^24
// in magnitude -- (L+1) products of at most 128 * 64 per k, or 128^2 for
// L = 0 -- so its FP32 accumulation in TMEM is exact; levels 6 and 7 carry
// weights 2^-56 and 2^-63 and their FP32 rounding is far below FP64 rounding.
// Longer K runs in passes of 512, each with its own scales and one rounding,
// that accumulate into C in FP64 (up to four passes in a launch).  One scale for
// four passes would save that accumulation, but an element then keeps fewer
// bits wherever its row is larger in another pass: rows that are large in
// opposite passes (a factor 1e11) lost half of their digits.
//
// Tensor-core layout.  Output tile 128 x 64.  The eight digit planes of the
// column operand are stacked along N in shared memory (plane t = rows
// 64 t .. 64 t + 63), so one MMA per row digit s covers every column digit
// t <= 7 - s at once: D columns [64 s, 512) receive A_s B_t into level block
// s + t.  TMEM holds the eight level blocks (512 columns); an MMA wider than
// 256 columns is issued as two, reusing A through the collector buffer.
//
// Recombination (epilogue, per element): the exact levels 0..5 in a 64-bit
// integer and levels 6..7 in FP32; one rounding to FP64, in integer
// instructions.  TMEM holds one set of level blocks, so the MMAs wait while a
// pass's sums are read: that part is only conversion and integer multiply-adds
// (about 25 instructions per element, eight warps), and the normalisation,
// scaling, accumulation (FP64 adds, C in L2) and stores run under the MMAs of the
// next pass or tile.
//
// CTA = 10 warps, persistent, one CTA per SM, output tiles assigned round
// robin: warp 0 bulk-copies the digit planes (two stages of 96 KB: 8 row
// planes of 128 x 32 and 8 column planes of 64 x 32, each a 64-byte-swizzled
// shared-memory image), warp 1 owns TMEM and issues the MMAs, warps 2..9
// read TMEM and write C.  Every wait is bounded.
//
// Bound by the tensor pipe: 36 BF16 products per FP64 product, 53 TFLOP/s at
// the measured cuBLAS BF16 rate.  Measured, kernel alone: 4096 x 32768 x 2048
// 10.4 ms (52.6 TFLOP/s; 17.5 ms with four epilogue warps that converted
// through the FP64 pipe before they released TMEM), 4096 x 4096 x 512 0.344 ms
// (0.526), 1520^3 0.156 ms (0.266).
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "dgemm_tc.h"
#include "tc_common.cuh"

namespace corr {

namespace {

constexpr int DS = 8;                     // digit planes per operand
constexpr int TM = 128;                   // output tile rows
constexpr int TN = kDgColTile;            // output tile columns
constexpr int DKB = 32;                   // K per stage: 64-byte tile rows
constexpr int KPASS = 512;                // K per pass (exact levels 0..5)
constexpr int KCHUNK = 2048;              // K per launch (digit planes in the workspace)
constexpr int PASS_KB = KPASS / DKB;
constexpr int PASSES = KCHUNK / KPASS;    // scales per row and launch
constexpr int A_PLANE = TM * DKB * 2;     // 8 KB
constexpr int B_PLANE = TN * DKB * 2;     // 4 KB
constexpr int A_BYTES = DS * A_PLANE;     // 64 KB
constexpr int STAGE = A_BYTES + DS * B_PLANE;  // 96 KB
constexpr int NSTAGE = 2;
constexpr int EWARPS = 8;                 // epilogue warps: two per TMEM lane quarter
constexpr int ECOLS = TN / (EWARPS / 4);  // columns of an epilogue warp
constexpr int NTHREADS = 64 + 32 * EWARPS;
constexpr uint32_t SW64 = 4;              // descriptor layout type: 64-byte swizzle
constexpr uint32_t TMEM_COLS = 512;

// Element offset of (row rr, k kk) inside one TR x 32 plane image: 16-byte
// chunk c of row rr sits at chunk c ^ ((rr >> 1) & 3).
__host__ __device__ inline int plane_offset(int rr, int kk) {
  return rr * DKB + ((((kk >> 3) ^ (rr >> 1)) & 3) << 3) + (kk & 7);
}

__device__ __forceinline__ long long view_row(const MatView& v, long long r) {
  return (r / v.rdiv) * v.rs_hi + (r % v.rdiv) * v.rs_lo;
}

// ---------------------------------------------------------------- slicing
// The largest biased exponent of each row in a pass, em[pass][r] (0 for a row
// without a normal value: all digits zero).  |x| < 2^(em - 1022) over the row.
__device__ __forceinline__ int row_scale(int em) { return em > 0 ? em - 1022 : 0; }
__device__ __forceinline__ int biased_exponent(double x) {
  return (__double2hiint(x) >> 20) & 0x7FF;
}
// Nonzero exactly when x is not +-0.
__device__ __forceinline__ uint32_t nonzero_bits(double x) {
  return ((uint32_t)__double2hiint(x) << 1) | (uint32_t)__double2loint(x);
}
// Rows the splitting cannot represent: not finite, or so small that the digits
// would lose subnormal elements.
__device__ __forceinline__ bool row_out_of_range(int em, uint32_t nz) {
  return em == 0x7FF || (em < 64 && nz != 0);
}

// The eight digits of x / 2^er as FP32 integers, most significant first.
__device__ __forceinline__ void digits_of(double x, int er, float (&d)[DS]) {
  const int hi = __double2hiint(x);
  const int E = (hi >> 20) & 0x7FF;
  unsigned long long H = 0;  // round(|x| 2^(56 - er)) <= 2^56
  if (E > 0) {
    const unsigned long long m =
        ((unsigned long long)((hi & 0xFFFFF) | 0x100000) << 32) | (uint32_t)__double2loint(x);
    const int t = E - 1019 - er;  // <= 3
    if (t >= 0) H = m << t;
    else if (t > -54) H = (m + (1ull << (-t - 1))) >> (-t);
  }
  // balanced digits: add 64 at each of the seven low base-128 positions, then
  // digit = (7-bit field) - 64; the sign of x in the one FMA that converts a
  // field (bits of 2^23 + field) to the signed digit, exactly
  constexpr unsigned long long BIAS = 0x40ull | (0x40ull << 7) | (0x40ull << 14) |
                                      (0x40ull << 21) | (0x40ull << 28) | (0x40ull << 35) |
                                      (0x40ull << 42);
  const unsigned long long Hb = H + BIAS;
  const float sg = hi < 0 ? -1.f : 1.f;
  const float c64 = -8388672.0f * sg, c0 = -8388608.0f * sg;
  const uint32_t w0 = (uint32_t)Hb, w1 = (uint32_t)(Hb >> 28), w2 = (uint32_t)(Hb >> 49);
#pragma unroll
  for (int p = 0; p < 7; ++p) {
    const uint32_t u = ((p < 4 ? w0 >> (7 * p) : w1 >> (7 * (p - 4))) & 127u) | 0x4B000000u;
    d[DS - 1 - p] = fmaf(__uint_as_float(u), sg, c64);
  }
  d[0] = fmaf(__uint_as_float(w2 | 0x4B000000u), sg, c0);  // 0 .. 128
}
// Two small integers (exact in BF16) packed as BF16, the first in the low half.
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}

// Eight consecutive k of one row -> eight 16-byte chunks, one per plane.
template <int TR>
__device__ __forceinline__ void store_chunk(const double (&x)[8], int er, uint16_t* dst) {
  uint32_t w[DS][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a[DS], b[DS];
    digits_of(x[2 * j], er, a);
    digits_of(x[2 * j + 1], er, b);
#pragma unroll
    for (int s = 0; s < DS; ++s) w[s][j] = pack_bf16(a[s], b[s]);
  }
#pragma unroll
  for (int s = 0; s < DS; ++s)
    *reinterpret_cast<uint4*>(dst + (size_t)s * (TR * DKB)) =
        make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
}

// The arrival counters of a product whose tiles are split over K start at zero;
// the slicing of its row operand, just ahead of it, clears them.
__device__ __forceinline__ void clear_tickets(unsigned* zero, int n) {
  if (blockIdx.y) return;
  for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < n; x += gridDim.x * blockDim.x)
    zero[x] = 0u;
}

// Slicing of an operand whose k are adjacent in memory: `lpr` lanes (a power
// of two) take one row's part of one pass (blockIdx.y), find its exponent and
// write its digit planes in one launch; the second read comes from L1/L2.  Bound by HBM (8 bytes
// read, 16 written per element).  Tile images [rt][kb][s] of TR x 32, zero
// beyond rows and kn; e[pass][rows_pad].
template <int TR>
__global__ void __launch_bounds__(256) slice_krow_kernel(MatView v, long long r0, int rows,
                                                         int rows_pad, int k0,
                                                         int kn, int nkb, int lpr,
                                                         int* __restrict__ e,
                                                         uint16_t* __restrict__ out,
                                                         int* __restrict__ status,
                                                         unsigned* __restrict__ zero, int nzero) {
  clear_tickets(zero, nzero);
  const int lane = threadIdx.x & 31, sub = lane & (lpr - 1), per = 32 / lpr;
  const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
  const int b0 = blockIdx.y * PASS_KB;                   // the pass's first K block,
  const int nch = min(PASS_KB, nkb - b0) * (DKB / 8);    // its chunks of 8 k
  kn = min(KPASS, kn - b0 * DKB);                        // and its k
  for (long long g = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
       g * per < rows_pad; g += nwarp) {
    const long long r = g * per + lane / lpr;  // below rows_pad, a multiple of per
    const bool live = r < rows;
    const double* p = live ? v.p + view_row(v, r0 + r) + (k0 + b0 * DKB) : nullptr;
    int em = 0;
    uint32_t nz = 0;
    if (live)
      for (int k = sub; k < kn; k += lpr) {
        const double x = p[k];
        em = max(em, biased_exponent(x));
        nz |= nonzero_bits(x);
      }
    for (int o = lpr >> 1; o > 0; o >>= 1) {
      em = max(em, __shfl_xor_sync(0xffffffffu, em, o));
      nz |= __shfl_xor_sync(0xffffffffu, nz, o);
    }
    if (sub == 0) {
      e[(size_t)blockIdx.y * rows_pad + r] = em;
      if (status && row_out_of_range(em, nz)) atomicOr(status, kStatusNeedFp64);
    }
    const int er = row_scale(em);
    const int rt = (int)(r / TR), rr = (int)(r % TR);
    uint16_t* row = out + ((size_t)rt * nkb + b0) * DS * (TR * DKB);
    const bool vec = (reinterpret_cast<uintptr_t>(p) & 15) == 0;
    for (int kc = sub; kc < nch; kc += lpr) {
      double x[8];
      const int k = kc * 8;
      if (live && vec && k + 8 <= kn) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double2 t = *reinterpret_cast<const double2*>(p + k + 2 * j);
          x[2 * j] = t.x;
          x[2 * j + 1] = t.y;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = live && k + j < kn ? p[k + j] : 0.0;
      }
      store_chunk<TR>(x, er,
                      row + (size_t)(kc >> 2) * DS * (TR * DKB) + plane_offset(rr, (kc & 3) * 8));
    }
  }
}

// Operands whose rows are adjacent in memory (k strided): exponents first,
// one lane per row and eight warps over the k of a block's segment (blockIdx.y),
// combined by a maximum in shared and global memory (e zeroed before), ...
constexpr int kExpSeg = 256;
static_assert(KPASS % kExpSeg == 0, "a segment lies in one pass");
__global__ void __launch_bounds__(256) col_exponent_kernel(MatView v, long long r0, int rows,
                                                           int rows_pad, int k0, int kn,
                                                           int* __restrict__ e,
                                                           int* __restrict__ status) {
  __shared__ int sm[8][32];
  __shared__ uint32_t snz[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long r = blockIdx.x * 32ll + lane;
  const int kb = blockIdx.y * kExpSeg, ke = min(kn, kb + kExpSeg);
  int em = 0;
  uint32_t nz = 0;
  if (r < rows) {
    const double* p = v.p + view_row(v, r0 + r) + (long long)k0 * v.ks;
#pragma unroll 8
    for (int k = kb + w; k < ke; k += 8) {
      const double x = p[(long long)k * v.ks];
      em = max(em, biased_exponent(x));
      nz |= nonzero_bits(x);
    }
  }
  sm[w][lane] = em;
  snz[w][lane] = nz;
  __syncthreads();
  if (w == 0 && r < rows) {
#pragma unroll
    for (int q = 1; q < 8; ++q) {
      em = max(em, sm[q][lane]);
      nz |= snz[q][lane];
    }
    atomicMax(&e[(size_t)(kb / KPASS) * rows_pad + r], em);
    // per segment of k: a small segment of a large row also takes the FP64 pipe
    if (status && row_out_of_range(em, nz)) atomicOr(status, kStatusNeedFp64);
  }
}

// ... then the digits: one thread per (row, 16 k), consecutive threads on
// consecutive rows; the two 16-byte chunks of a plane it writes fill one
// 32-byte sector of the swizzled image.
template <int TR>
__global__ void __launch_bounds__(256) slice_kcol_kernel(MatView v, long long r0, int rows,
                                                         int rows_pad, int k0,
                                                         int kn, int nkb,
                                                         const int* __restrict__ e,
                                                         uint16_t* __restrict__ out,
                                                         unsigned* __restrict__ zero, int nzero) {
  clear_tickets(zero, nzero);
  const int nc2 = nkb * (DKB / 16);
  const long long total = (long long)rows_pad * nc2;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const long long r = t % rows_pad;
    const int kc2 = (int)(t / rows_pad);
    const bool live = r < rows;
    const int er = row_scale(e[(size_t)(kc2 / (KPASS / 16)) * rows_pad + r]);
    const double* p = live ? v.p + view_row(v, r0 + r) + (long long)k0 * v.ks : nullptr;
    const int rt = (int)(r / TR), rr = (int)(r % TR);
    uint16_t* tile = out + ((size_t)rt * nkb + (kc2 >> 1)) * DS * (TR * DKB);
    double x[2][8];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int k = kc2 * 16 + j;
      x[j >> 3][j & 7] = live && k < kn ? p[(long long)k * v.ks] : 0.0;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
      store_chunk<TR>(x[h], er, tile + plane_offset(rr, (kc2 & 1) * 16 + h * 8));
  }
}

// ---------------------------------------------------------------- product
struct DgArgs {
  const uint16_t* Ad;  // row-operand digit tiles [mt][kb][s] (128 x 32)
  const uint16_t* Bd;  // column-operand digit tiles [nt][kb][s] (64 x 32)
  const int* ea;       // row exponents [pass][lea]
  const int* eb;       // column exponents [pass][leb]
  int lea, leb;
  OutView C;
  double alpha;        // applied when `scaled`; else alpha = +-2^alpha_exp, its sign bit in `sign`
  int alpha_exp, scaled;
  uint32_t sign;
  int M, N, nkb, mtn, ntn;  // M: end of this launch's rows (m0 its first)
  int m0;
  int col_major_order;  // units nt-major (shared column tile adjacent)
  int a_lower, k0, accumulate;
  int nsplit, kper;  // parts of a tile's K blocks (kper each): units are (tile, part)
  int nslot;         // nsplit > 1: [tile][slot][warp][column][lane] sums, slot = part + pass,
  unsigned long long* part_hi;
  float* part_tail;
  unsigned* ticket;  // per (tile, pass, warp) the parts, per (tile, warp) the passes that arrived
  int tiles;
  long long total;
};

struct DgCtl {
  uint64_t full[NSTAGE];
  uint64_t empty[NSTAGE];
  uint64_t afull;
  uint64_t aempty;
  uint64_t fin;
  uint32_t tmem;
  int abort;
};

// Unit u: its tile, and the part of its K blocks.
template <bool SPLIT>
__device__ __forceinline__ void unit_tile(const DgArgs& a, long long u, int* mt, int* nt) {
  if (SPLIT) u /= a.nsplit;
  if (a.col_major_order) {
    *nt = (int)(u / a.mtn);
    *mt = (int)(u % a.mtn);
  } else {
    *mt = (int)(u / a.ntn);
    *nt = (int)(u % a.ntn);
  }
}

// K blocks of this launch that tile row mt needs (lower-triangular A: k <= m).
__device__ __forceinline__ int unit_kblocks(const DgArgs& a, int mt) {
  if (!a.a_lower) return a.nkb;
  const int kend = a.m0 + (mt + 1) * TM - a.k0;  // local k < kend can be nonzero
  return kend <= 0 ? 0 : min(a.nkb, (kend + DKB - 1) / DKB);
}

// K blocks [*kb0, *kb1) of unit u (empty past a triangular tile's last block).
template <bool SPLIT>
__device__ __forceinline__ void unit_range(const DgArgs& a, long long u, int mt, int* kb0,
                                           int* kb1) {
  const int n = unit_kblocks(a, mt);
  *kb0 = SPLIT ? (int)(u % a.nsplit) * a.kper : 0;
  *kb1 = SPLIT ? min(n, *kb0 + a.kper) : n;
}

// Sums of one output element over a pass: levels 0..5 as an exact 64-bit integer
// in level-5 units (2^-49 of the row and column scales; |sum| <= 2^58) and levels
// 6..7 in FP32 level-5 units.
struct ElemSum {
  unsigned long long hi;
  float tail;
};
// Bits of 2^23 + 2^22 (FP32): adding it to an integer |x| <= 2^22 leaves x in
// the low bits (a conversion on the FP32 pipe; F2I runs at a quarter rate or
// less); the constants come off together.
constexpr uint32_t kMagicBits = 0x4B400000u;
constexpr float kMagic = 12582912.0f;
constexpr unsigned long long kMagicSum =
    (unsigned long long)kMagicBits *
    (1ull + (1ull << 7) + (1ull << 14) + (1ull << 21) + (1ull << 28) + (1ull << 35));

template <bool WIDE>
__device__ __forceinline__ ElemSum combine_levels(const float (&x)[DS]) {
  int u[6];
#pragma unroll
  for (int L = 0; L < 6; ++L)
    u[L] = WIDE ? __float2int_rn(x[L]) + (int)kMagicBits : __float_as_int(x[L] + kMagic);
  unsigned long long v = (unsigned long long)(long long)u[5] - kMagicSum;
  v += (unsigned long long)((long long)u[4] * (1 << 7));
  v += (unsigned long long)((long long)u[3] * (1 << 14));
  v += (unsigned long long)((long long)u[2] * (1 << 21));
  v += (unsigned long long)((long long)u[1] * (1 << 28));
  v += (unsigned long long)(uint32_t)(u[0] << 3) << 32;  // u0 2^35 modulo 2^64
  return ElemSum{v, fmaf(x[7], 0.0078125f, x[6]) * 0.0078125f};
}

template <bool WIDE>
__device__ __forceinline__ void combine_chunk(ElemSum* sum, const float (&lv)[DS][8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    float x[DS];
#pragma unroll
    for (int L = 0; L < DS; ++L) x[L] = lv[L][e];
    sum[e] = combine_levels<WIDE>(x);
  }
}

// The FP64 value 2^sh (hi + tail), hi in level-5 units, rounded once to nearest
// even.  32-bit integer and FP32 instructions throughout: this GPU's FP64 pipe
// takes two lanes per clock per SM, so one FP64 instruction per element --
// a 64-bit conversion, a multiply by alpha = 1, a negation -- is 2 us of a tile.
// tail goes in at 2^-11 of a level-5 unit (2^-60 of the scales), fewer bits
// when hi is that large.  No branches, so that eight elements overlap; *odd is
// set for a value at the ends of the exponent range (finish_slow).
__device__ __forceinline__ unsigned long long finish_sum(long long hi, float tail, int sh,
                                                         uint32_t sign, bool* odd) {
  const int hh = (int)(hi >> 32);
  const int n = min(11, __clz(hh ^ (hh >> 31)) - 2);  // hi << n within 2^62; |hi| < 2^61
  const long long V = (hi << n) + (__float2int_rn(tail * 2048.f) >> (11 - n));  // |tail| < 2^20
  const unsigned long long a = (unsigned long long)(V < 0 ? -V : V);
  const int lz = __clzll((long long)a) & 63;
  const unsigned long long m = a << lz;  // top bit set; value = m 2^(sh - n - lz)
  const int ex = sh - n - lz + 1086;     // biased exponent of the top bit
  const uint32_t rem = (uint32_t)m & 0x7FFu;
  unsigned long long b = m >> 11;
  b += (rem + (uint32_t)(b & 1)) > 0x400u ? 1 : 0;  // to nearest even; a carry moves up
  b += (unsigned long long)(uint32_t)(ex - 1) << 52;
  const bool zero = a == 0;
  *odd = !zero && (ex <= 0 || ex >= 2046);
  b |= (unsigned long long)(sign ^ (V < 0 ? 0x80000000u : 0u)) << 32;
  return zero ? 0ull : b;
}

// The same at the ends of the exponent range: subnormal, or near the largest.
__device__ __noinline__ double finish_slow(long long hi, float tail, int sh, uint32_t sign) {
  const int hh = (int)(hi >> 32);
  const int n = min(11, __clz(hh ^ (hh >> 31)) - 2);
  const long long V = (hi << n) + (__float2int_rn(tail * 2048.f) >> (11 - n));
  const double r = ldexp((double)V, sh - n);
  return sign ? -r : r;
}

// SPLIT: tiles split over K (nsplit > 1); a kernel of its own, since its exchange
// costs the other one registers (3 % at K above 512).
template <bool SPLIT>
__global__ void __launch_bounds__(NTHREADS, 1) dgemm_tc_kernel(DgArgs a, int* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* tiles = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  DgCtl* ctl = reinterpret_cast<DgCtl*>(tiles + NSTAGE * STAGE);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
    }
    mbar_init(&ctl->afull, 1);
    mbar_init(&ctl->aempty, EWARPS);
    mbar_init(&ctl->fin, 1);
    ctl->abort = 0;
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(&ctl->tmem, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl->tmem;
  volatile int* abort = &ctl->abort;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    int st = 0;
    uint32_t ph = 0;
    uint32_t last_ph[NSTAGE];
    bool has[NSTAGE];
    for (int s = 0; s < NSTAGE; ++s) has[s] = false;
    bool ok = true;
    for (long long u = blockIdx.x; u < a.total && ok; u += gridDim.x) {
      int mt, nt;
      unit_tile<SPLIT>(a, u, &mt, &nt);
      int kb0, kb1;
      unit_range<SPLIT>(a, u, mt, &kb0, &kb1);
      for (int kb = kb0; kb < kb1; ++kb) {
        bool got = true;
        if (lane == 0) got = mbar_wait(&ctl->empty[st], ph ^ 1, abort, status);
        if (!__shfl_sync(0xffffffffu, got ? 1 : 0, 0)) {
          ok = false;
          break;
        }
        uint64_t* bar = &ctl->full[st];
        if (lane == 0) mbar_expect_tx(bar, STAGE);
        __syncwarp();
        uint8_t* sb = tiles + (size_t)st * STAGE;
        if (lane < DS)
          bulk_load(sb + lane * A_PLANE,
                    a.Ad + (((size_t)mt * a.nkb + kb) * DS + lane) * (TM * DKB), A_PLANE, bar);
        else if (lane < 2 * DS)
          bulk_load(sb + A_BYTES + (lane - DS) * B_PLANE,
                    a.Bd + (((size_t)nt * a.nkb + kb) * DS + (lane - DS)) * (TN * DKB), B_PLANE,
                    bar);
        has[st] = true;
        last_ph[st] = ph;
        if (++st == NSTAGE) {
          st = 0;
          ph ^= 1;
        }
      }
    }
    if (lane == 0) {  // never leave with a copy still landing in shared memory
      int never = 0;
      for (int s = 0; s < NSTAGE; ++s)
        if (has[s]) mbar_wait(&ctl->full[s], last_ph[s], &never, status);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int st = 0;
      uint32_t ph = 0, nuse = 0;
      bool ok = true;
      uint32_t idn[5];  // instruction descriptors for N = 64 k, k = 1..4
      for (int k = 1; k <= 4; ++k) idn[k] = idesc_f16(1u, TM, 64u * k);
      const uint64_t dbase = smem_desc(smem_u32(tiles), 16, 512, SW64);
      for (long long u = blockIdx.x; u < a.total && ok; u += gridDim.x) {
        int mt, nt;
        unit_tile<SPLIT>(a, u, &mt, &nt);
        int kb0, kb1;
        unit_range<SPLIT>(a, u, mt, &kb0, &kb1);
        if (kb1 <= kb0) continue;
        if (!mbar_wait(&ctl->aempty, (nuse & 1) ^ 1, abort, status)) break;
        tc_fence_after();
        for (int kb = kb0; kb < kb1; ++kb) {
          const bool first = kb == kb0 || kb % PASS_KB == 0;
          if (first && kb != kb0) {  // next K pass: the epilogue takes the sums first
            tc_commit(&ctl->afull);
            ++nuse;
            if (!mbar_wait(&ctl->aempty, (nuse & 1) ^ 1, abort, status)) {
              ok = false;
              break;
            }
            tc_fence_after();
          }
          if (!mbar_wait(&ctl->full[st], ph, abort, status)) {
            ok = false;
            break;
          }
          const uint64_t ds = dbase + (uint64_t)(((uint32_t)st * STAGE) >> 4);
#pragma unroll
          for (int kk = 0; kk < DKB / 16; ++kk) {
            const uint64_t bq = ds + (uint64_t)((A_BYTES + kk * 32) >> 4);
#pragma unroll
            for (int s = 0; s < DS; ++s) {
              const uint64_t ar = ds + (uint64_t)((s * A_PLANE + kk * 32) >> 4);
              const uint32_t acc = !first || kk || s ? 1u : 0u;
              const uint32_t d = tmem + 64u * s;
              const int nblk = DS - s;  // column planes 0 .. 7 - s
              if (nblk > 4) {
                tc_mma_f16_ca<0>(d, ar, bq, idn[4], acc);
                tc_mma_f16_ca<2>(d + 256u, ar, bq + (uint64_t)((4 * B_PLANE) >> 4),
                                 idn[nblk - 4], acc);
              } else {
                tc_mma_f16(d, ar, bq, idn[nblk], acc);
              }
            }
          }
          tc_commit(&ctl->empty[st]);
          if (++st == NSTAGE) {
            st = 0;
            ph ^= 1;
          }
        }
        if (ok) tc_commit(&ctl->afull);
        ++nuse;
      }
      tc_commit(&ctl->fin);
      int never = 0;
      mbar_wait(&ctl->fin, 0, &never, status);
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3;              // TMEM lane quarter of this warp
    const int c0 = ((warp - 2) >> 2) * ECOLS;  // its columns of the tile
    const int arow = 32 * q + lane;
    const uint32_t tq = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)c0;
    uint32_t nuse = 0;
    bool ok = true;
    for (long long u = blockIdx.x; u < a.total && ok; u += gridDim.x) {
      int mt, nt;
      unit_tile<SPLIT>(a, u, &mt, &nt);
      int kb0, kb1;
      unit_range<SPLIT>(a, u, mt, &kb0, &kb1);
      if (kb1 <= kb0) continue;
      const int pass1 = (kb1 - 1) / PASS_KB;
      for (int pass = kb0 / PASS_KB; pass <= pass1; ++pass, ++nuse) {
        const bool got = mbar_wait(&ctl->afull, nuse & 1, abort, status);
        if (!__all_sync(0xffffffffu, got)) {
          ok = false;
          break;
        }
        tc_fence_after();
        // only this part holds the MMAs of the next pass up: sums into
        // registers, then the accumulators go back
        ElemSum sum[ECOLS];
#pragma unroll
        for (int c = 0; c < ECOLS / 8; ++c) {
          float lv[DS][8];
#pragma unroll
          for (int L = 0; L < DS; ++L) tmem_ld8(tq + (uint32_t)(TN * L + 8 * c), lv[L]);
          tc_wait_ld();
#pragma unroll
          for (int L = 0; L < DS; ++L) ld_ready<8>(lv[L]);
          float mx = 0.f;
#pragma unroll
          for (int e = 0; e < 8; ++e)
#pragma unroll
            for (int L = 0; L < 6; ++L) mx = fmaxf(mx, fabsf(lv[L][e]));
          if (__any_sync(0xffffffffu, mx > 4194304.f))
            combine_chunk<true>(sum + 8 * c, lv);
          else
            combine_chunk<false>(sum + 8 * c, lv);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->aempty);
        // A part of the tile's K: the warp leaves its sums in L2, and the warp that
        // arrives last adds the parts of the pass up (integers exactly, the FP32
        // tails in part order) and rounds; with several passes it leaves the result
        // in L2 again, and the last of those adds the passes up in their order.  No
        // warp waits for another.
        const long long tile = SPLIT ? u / a.nsplit : u;
        auto slot = [&](int part, int ps) {
          return ((size_t)(tile * a.nslot + part + ps) * EWARPS + (warp - 2)) * ECOLS * 32 + lane;
        };
        auto arrive_last = [&](long long t, int count) -> bool {
          __threadfence();
          __syncwarp();
          unsigned n = 0;
          if (lane == 0) n = atomicAdd(&a.ticket[t * EWARPS + (warp - 2)], 1u);
          const bool last = __shfl_sync(0xffffffffu, n, 0) == (unsigned)count - 1;
          __threadfence();
          return last;
        };
        const int kblocks = SPLIT ? unit_kblocks(a, mt) : 0;
        const int q0 = SPLIT ? pass * PASS_KB / a.kper : 0;
        const bool apart = SPLIT && kblocks > PASS_KB;  // passes added up at the end
        if (SPLIT) {
          const size_t mine = slot((int)(u - tile * a.nsplit), pass);
#pragma unroll
          for (int e = 0; e < ECOLS; ++e) {
            __stcg(&a.part_hi[mine + 32 * e], sum[e].hi);
            __stcg(&a.part_tail[mine + 32 * e], sum[e].tail);
          }
          const int parts = (min(kblocks, (pass + 1) * PASS_KB) - 1) / a.kper - q0 + 1;
          if (!arrive_last(tile * PASSES + pass, parts)) continue;
#pragma unroll
          for (int e = 0; e < ECOLS; ++e) sum[e] = ElemSum{0ull, 0.f};
          for (int q = 0; q < parts; ++q) {
            const size_t at = slot(q0 + q, pass);
#pragma unroll
            for (int e = 0; e < ECOLS; ++e) {
              sum[e].hi += __ldcg(&a.part_hi[at + 32 * e]);
              sum[e].tail += __ldcg(&a.part_tail[at + 32 * e]);
            }
          }
        }
        const long long m = a.m0 + (long long)mt * TM + arow;
        const bool mlive = m < a.M;
        const int n0 = nt * TN + c0;
        double* dst = a.C.p + (m / a.C.rdiv) * a.C.rs_hi + (m % a.C.rdiv) * a.C.rs_lo +
                      (long long)n0 * a.C.cs;
        const bool vec = a.C.cs == 1 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
        // columns c .. c + 7 of this lane's row; all loads before the first add or store
        auto put = [&](int c, double (&r)[8], bool accumulate) {
          const int live = mlive ? min(8, a.N - n0 - c) : 0;
          const bool wide = vec && live == 8;
          double* d = dst + (long long)c * a.C.cs;
          double2* d2 = reinterpret_cast<double2*>(d);
          if (accumulate) {
            double o[8];
            if (wide) {
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const double2 t = d2[e];
                o[2 * e] = t.x;
                o[2 * e + 1] = t.y;
              }
            } else {
#pragma unroll
              for (int e = 0; e < 8; ++e) o[e] = e < live ? d[(long long)e * a.C.cs] : 0.0;
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) r[e] += o[e];
          }
          if (wide) {
#pragma unroll
            for (int e = 0; e < 4; ++e) d2[e] = make_double2(r[2 * e], r[2 * e + 1]);
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (e < live) d[(long long)e * a.C.cs] = r[e];
          }
        };
        // Normalise and store, eight columns per step: a rolled loop that moves
        // the remaining sums down the register array (unrolled over 32 columns the
        // code ran at the rate of its instruction fetches).
        const int em = (mlive ? row_scale(a.ea[(size_t)pass * a.lea + (m - a.m0)]) : 0) +
                       a.alpha_exp - 49;
        const int en = row_scale(a.eb[(size_t)pass * a.leb + n0 + lane]);
        const size_t rounded = slot(q0, pass);
#pragma unroll 1
        for (int c = 0; c < ECOLS; c += 8) {
          double r[8];
          uint32_t odd = 0;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            bool x;
            r[e] = __longlong_as_double((long long)finish_sum(
                (long long)sum[e].hi, sum[e].tail,
                em + __shfl_sync(0xffffffffu, en, c + e), a.sign, &x));
            odd |= x ? 1u << e : 0u;
          }
          if (__any_sync(0xffffffffu, odd != 0)) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const int sh = em + __shfl_sync(0xffffffffu, en, c + e);
              if (odd >> e & 1)
                r[e] = finish_slow((long long)sum[e].hi, sum[e].tail, sh, a.sign);
            }
          }
          if (a.scaled) {
#pragma unroll
            for (int e = 0; e < 8; ++e) r[e] *= a.alpha;
          }
          if (apart) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              __stcg(&a.part_hi[rounded + 32 * (c + e)],
                     (unsigned long long)__double_as_longlong(r[e]));
          } else {
            put(c, r, a.accumulate || pass > 0);
          }
#pragma unroll
          for (int e = 0; e + 8 < ECOLS; ++e) sum[e] = sum[e + 8];
        }
        if (apart) {
          const int passes = (kblocks + PASS_KB - 1) / PASS_KB;
          if (!arrive_last((long long)a.tiles * PASSES + tile, passes)) continue;
#pragma unroll 1
          for (int c = 0; c < ECOLS; c += 8) {
            double r[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) r[e] = 0.0;
#pragma unroll 2
            for (int p = 0; p < passes; ++p) {
              const size_t at = slot(p * PASS_KB / a.kper, p) + 32 * c;
#pragma unroll
              for (int e = 0; e < 8; ++e)
                r[e] += __longlong_as_double((long long)__ldcg(&a.part_hi[at + 32 * e]));
            }
            put(c, r, a.accumulate);
          }
        }
      }
      if (!ok) break;
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

constexpr size_t kDgSmem = (size_t)NSTAGE * STAGE + sizeof(DgCtl) + 1024;
static_assert(kDgSmem <= 227 * 1024, "shared memory");

int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }
size_t align256(size_t b) { return (b + 255) / 256 * 256; }

template <int TR>
int slice_operand(corr_context* c, const MatView& v, long long r0, int rows, int rows_pad, int k0, int kn,
                  int nkb, int* e, uint16_t* out, unsigned* zero = nullptr, int nzero = 0) {
  const int cap = c->sms * 16;
  int* status = c->digit_guard ? &c->dres->status : nullptr;
  if (v.ks == 1) {  // k contiguous
    int lpr = 1;
    while (lpr < 32 && lpr < nkb * (DKB / 8)) lpr *= 2;
    const dim3 grid((unsigned)std::min(ceil_div((long long)rows_pad * lpr, 256), cap),
                    (unsigned)ceil_div(nkb, PASS_KB));
    slice_krow_kernel<TR><<<grid, 256, 0, c->stream>>>(v, r0, rows, rows_pad, k0, kn, nkb, lpr, e,
                                                       out, status, zero, nzero);
    CORR_CUDA(cudaGetLastError());
    c->launches += 1;
    return CORR_OK;
  }
  CORR_CUDA(cudaMemsetAsync(e, 0, (size_t)rows_pad * 4 * ceil_div(kn, KPASS), c->stream));
  const dim3 eg((unsigned)ceil_div(rows, 32), (unsigned)ceil_div(kn, kExpSeg));
  col_exponent_kernel<<<eg, 256, 0, c->stream>>>(v, r0, rows, rows_pad, k0, kn, e, status);
  CORR_CUDA(cudaGetLastError());
  const int grid = std::min(ceil_div((long long)rows_pad * nkb * (DKB / 16), 256), cap);
  slice_kcol_kernel<TR><<<grid, 256, 0, c->stream>>>(v, r0, rows, rows_pad, k0, kn, nkb, e, out, zero,
                                                      nzero);
  CORR_CUDA(cudaGetLastError());
  c->launches += 2;
  return CORR_OK;
}

}  // namespace

// Parts of each tile's K blocks: few tiles (or a last wave that is nearly
// empty) leave SMs idle, so the tiles of one launch may be split over K.  The
// cheapest number of parts, counting a K block of 2304 tensor clocks, 3000 for
// taking a pass's sums out of TMEM, and for split tiles about 6000 more for the
// exchange through L2.  715^3 (72 tiles): 39 us with two parts, 48 us whole.
constexpr int kSplitSms = 152;
constexpr int kMaxSplit = 16;
constexpr long long kMaxSplitSlots = 2 * kSplitSms;
static int k_parts(long long tiles, int nkb) {
  int best = 1;
  double cost = 0.0;
  for (int s = 1; s <= kMaxSplit && s <= nkb; ++s) {
    if (s > 1 && tiles * (s + ceil_div(nkb, PASS_KB) - 1) > kMaxSplitSlots) break;
    const int kper = ceil_div(nkb, s);
    int passes = 0;  // of the part that touches most
    for (int b = 0; b < nkb; b += kper)
      passes = std::max(passes, (std::min(nkb, b + kper) - 1) / PASS_KB - b / PASS_KB + 1);
    const double waves = (double)((tiles * s + kSplitSms - 1) / kSplitSms);
    const double t = waves * (kper * 2304.0 + 3000.0 * passes) + (s > 1 ? 6000.0 + 600.0 * s : 0.0);
    if (s == 1 || t < 0.95 * cost) {
      cost = t;
      best = s;
    }
  }
  return best;
}
// Sums and tickets of any split launch: 30 MB, part of every workspace (smaller
// products than the one a caller sized its workspace for may split further).
constexpr size_t kSplitBytes = (size_t)kMaxSplitSlots * TM * TN * 12 +
                               kMaxSplitSlots * (PASSES + 1) * EWARPS * 4;

// Rows (columns) of a launch for K (padded) of kp, a multiple of the tile: an
// operand's digit planes stay within kDgPlaneBytes (at least 256 tiles, so that a
// narrow product still fills the SMs).
static int plane_chunk(int rows, size_t kp, int tile) {
  const size_t fit = kDgPlaneBytes / (kp * DS * 2) / tile * tile;
  return (int)std::min<size_t>((size_t)ceil_div(rows, tile) * tile,
                               std::max<size_t>(fit, 256 * tile));
}

// Bytes of an operand's planes and exponents in any launch of plane_chunk(rows, kp,
// tile) rows; no less for a larger kp, so that a workspace also holds the products
// with a smaller K.
static size_t operand_bytes(int rows, size_t kp, int tile) {
  const size_t rp = (size_t)ceil_div(rows, tile) * tile, row = kp * DS * 2;
  const size_t planes = std::min(rp * row, std::max(kDgPlaneBytes, 256 * tile * row));
  // kp >= 32: an exponent per 512 of k is at most 1/64 of the planes
  const size_t exps = std::min(rp * 4 * ceil_div(kp, KPASS), planes / 64 + 4096);
  return align256(planes) + align256(exps);
}

size_t dgemm_tc_workspace(int M, int N, int K) {
  const size_t kp = (size_t)ceil_div(std::min(std::max(K, 1), KCHUNK), DKB) * DKB;
  return operand_bytes(M, kp, TM) + operand_bytes(N, kp, TN) + align256(kSplitBytes);
}

size_t dgemm_tc_columns_bytes(int rows, int K) {
  const size_t np = (size_t)ceil_div(rows, TN) * TN;
  const size_t kp = (size_t)ceil_div(std::max(K, 1), DKB) * DKB;
  return align256(np * kp * DS * 2) + align256(np * 4 * ceil_div(kp, KPASS));
}

int dgemm_tc_slice_columns(corr_context* c, const MatView& v, int rows, int K, void* ws,
                           DgColumns* out) {
  const int np = ceil_div(rows, TN) * TN;
  const size_t kp = (size_t)ceil_div(std::max(K, 1), DKB) * DKB;
  uint16_t* planes = static_cast<uint16_t*>(ws);
  int* e = reinterpret_cast<int*>(static_cast<uint8_t*>(ws) + align256(np * kp * DS * 2));
  for (int k0 = 0, p = 0; k0 < K; k0 += KCHUNK, ++p) {
    const int kn = std::min(KCHUNK, K - k0);
    CORR_TRY(slice_operand<TN>(c, v, 0, rows, np, k0, kn, ceil_div(kn, DKB), e + (size_t)p * PASSES * np,
                               planes + (size_t)p * KCHUNK * np * DS));
  }
  out->planes = planes;
  out->e = e;
  out->rows_pad = np;
  return CORR_OK;
}

int dgemm_tc(corr_context* c, const DgemmTc& g, void* ws) {
  if (g.M <= 0 || g.N <= 0) return CORR_OK;
  const size_t kp = (size_t)ceil_div(std::min(std::max(g.K, 1), KCHUNK), DKB) * DKB;
  const int mp = plane_chunk(g.M, kp, TM);
  const int np = g.pre ? ceil_div(g.N, TN) * TN : plane_chunk(g.N, kp, TN);
  uint8_t* w = static_cast<uint8_t*>(ws);
  uint16_t* Ad = reinterpret_cast<uint16_t*>(w);
  w += align256((size_t)mp * kp * DS * 2);
  int* ea = reinterpret_cast<int*>(w);
  const size_t passes = ceil_div(kp, KPASS);
  w += align256((size_t)mp * 4 * passes);
  uint16_t* Bw = reinterpret_cast<uint16_t*>(w);
  if (!g.pre) w += align256((size_t)np * kp * DS * 2);
  int* ebw = reinterpret_cast<int*>(w);
  if (!g.pre) w += align256((size_t)np * 4 * passes);
  static bool attr[64] = {};
  if (c->device < 0 || c->device >= 64 || !attr[c->device]) {
    for (auto k : {dgemm_tc_kernel<false>, dgemm_tc_kernel<true>})
      CORR_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kDgSmem));
    if (c->device >= 0 && c->device < 64) attr[c->device] = true;
  }
  const int chunks = std::max(1, ceil_div(g.K, KCHUNK));
  // alpha = +-2^x goes into the result's exponent and sign, exactly
  int ax = 0;
  const bool pow2 = std::frexp(std::fabs(g.alpha), &ax) == 0.5 && ax > -64 && ax < 64;
  for (int p = 0; p < chunks; ++p) {
    const int k0 = p * KCHUNK, kn = std::min(KCHUNK, g.K - k0);
    const int nkb = ceil_div(std::max(kn, 1), DKB);
    for (int n0 = 0; n0 < g.N; n0 += np) {
      const int cols = std::min(np, g.N - n0), ntn = ceil_div(cols, TN);
      const uint16_t* Bd = Bw;
      const int* eb = ebw;
      if (kn <= 0) {  // K == 0: zero digits give C = 0 (or C unchanged when accumulating)
        CORR_CUDA(cudaMemsetAsync(Bw, 0, (size_t)np * kp * DS * 2, c->stream));
        CORR_CUDA(cudaMemsetAsync(ebw, 0, (size_t)np * 4, c->stream));
      } else if (g.pre) {
        Bd = g.pre->planes +
             ((size_t)p * KCHUNK * g.pre->rows_pad + (size_t)g.col0 * nkb * DKB) * DS;
        eb = g.pre->e + (size_t)p * PASSES * g.pre->rows_pad + g.col0;
      } else {
        CORR_TRY(slice_operand<TN>(c, g.B, n0, cols, ntn * TN, k0, kn, nkb, ebw, Bw));
      }
      for (int m0 = 0; m0 < g.M; m0 += mp) {
        const int rows = std::min(mp, g.M - m0), mtn = ceil_div(rows, TM);
        const long long tiles = (long long)mtn * ntn;
        const int parts = mp >= g.M && np >= g.N && kn > 0 ? k_parts(tiles, nkb) : 1;
        unsigned long long* part_hi = reinterpret_cast<unsigned long long*>(w);
        float* part_tail = reinterpret_cast<float*>(part_hi + kMaxSplitSlots * TM * TN);
        unsigned* ticket = reinterpret_cast<unsigned*>(part_tail + kMaxSplitSlots * TM * TN);
        if (kn <= 0) {
          CORR_CUDA(cudaMemsetAsync(Ad, 0, (size_t)mp * kp * DS * 2, c->stream));
          CORR_CUDA(cudaMemsetAsync(ea, 0, (size_t)mp * 4, c->stream));
        } else if (n0 == 0 || mp < g.M) {  // else the planes of all rows are there
          CORR_TRY(slice_operand<TM>(c, g.A, m0, rows, mtn * TM, k0, kn, nkb, ea, Ad, ticket,
                                     parts > 1 ? (int)tiles * (PASSES + 1) * EWARPS : 0));
        }
        DgArgs a;
        a.Ad = Ad;
        a.Bd = Bd;
        a.ea = ea;
        a.eb = eb;
        a.lea = mtn * TM;
        a.leb = g.pre ? g.pre->rows_pad : ntn * TN;
        a.C = g.C;
        a.C.p += (long long)n0 * g.C.cs;
        a.alpha = g.alpha;
        a.scaled = pow2 ? 0 : 1;
        a.alpha_exp = pow2 ? ax - 1 : 0;
        a.sign = pow2 && g.alpha < 0.0 ? 0x80000000u : 0u;
        a.M = m0 + rows;
        a.N = cols;
        a.m0 = m0;
        a.nkb = nkb;
        a.mtn = mtn;
        a.ntn = ntn;
        // keep the larger operand's tile shared by adjacent units (L2 reuse)
        a.col_major_order = ntn * TN > mtn * TM ? 1 : 0;
        a.a_lower = g.a_lower ? 1 : 0;
        a.k0 = k0;
        a.accumulate = (g.accumulate || p > 0) ? 1 : 0;
        a.nsplit = parts;
        a.kper = ceil_div(nkb, parts);
        a.nslot = parts + ceil_div(nkb, PASS_KB) - 1;
        a.part_hi = part_hi;
        a.part_tail = part_tail;
        a.ticket = ticket;
        a.tiles = (int)tiles;
        a.total = tiles * a.nsplit;
        const int grid = (int)std::min<long long>(a.total, c->sms - c->spare_sms);
        (parts > 1 ? dgemm_tc_kernel<true> : dgemm_tc_kernel<false>)<<<grid, NTHREADS, kDgSmem,
                                                                    c->stream>>>(
            a, &c->dres->status);
        CORR_CUDA(cudaGetLastError());
        c->launches += 1;
      }
    }
  }
  return CORR_OK;
}

}  // namespace corr
