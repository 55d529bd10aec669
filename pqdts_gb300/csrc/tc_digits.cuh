// Banded products of FP64 operands on the tensor cores, by exact integer
// digits: the mixed path's gradient F^T.R (dL, pqdts.f90:975-1032) and its
// FP64-accurate objective checks F.X - P (L, 917-973).
//
// K, the dimension that a product sums over, is cut into groups of 256 (rows i
// of X, rows d of R).  The part of a row of F (or F^T) in a group, and the
// part of a column of X (or R), is scaled by a power of two of its own, so
// that its largest magnitude lies in [1/4, 1/2), rounded to 8 S = 56 bits and
// written as S = 7 signed digits in base 256, each exact in bf16:
//   x = 2^E (d_0 2^-8 + d_1 2^-16 + ... ),  |d_q| <= 128.
// A group's product is then a sum over digit pairs, and the pairs p + q = L of
// one level L share a weight 2^(-8 (L + 2)), so level L needs one integer sum
//   S_L = sum_k sum_{p + q = L} dF_p[k] dX_q[k]
// which the MMAs (bf16 in, FP32 accumulator in tensor memory) form exactly: a
// product of digits is at most 2^14, so a pair's sum over a group stays within
// 2^22 and the levels 0..3 within 2^24, the integers an FP32 accumulator
// holds; the next ones may pass that (by at most 1.75x, operands whose digits
// all have one sign) and then round by an ulp.  The levels 0 .. S - 1 are
// kept, 28 digit pairs.  After each group its sums are drained into a 64-bit
// integer at the larger of the two exponents (the sum's so far and the
// group's), so the error of an output is ~sqrt(K) 2^-58 of the largest of its
// groups' (row scale x column scale).
//
// Where the operands' magnitudes fall off steeply inside a group (the tails of
// a Poisson row against those of a detector's column), that can be more than
// a sum's own size allows: the double-FP32 kernels (k_fwd_df, k_trans_df) hold
// each operand to 48 bits of itself.  So the magnitudes are multiplied too, in
// bf16 (one more MMA a K slice), and an output whose sum of |f| |x| is too
// small beside its scales (dg_floor) is marked and left to those kernels,
// which skip all blocks without such an output.  So no entry is less accurate
// than they leave it, and most are more: relative to the sum of |F|^T |R|,
// gradient entries at M = 300 .. 6000 are off by 0.05-0.4 * 2^-48 at the
// median and 0.3-13 at the 99th percentile, by 2-7 and 12-65 in double-FP32
// alone (its own flushes below 2^-126 aside).  M = 10^4, N = 10^3: F.X 1.61 ms
// in digits and 0.14-0.60 for what they leave, F^T.R 1.58 and 0.09 (7.3-10.9
// and 8.9 in double-FP32), and 0.4 for the operands.  Iterates in the middle of
// a solve leave more, 20-40% of F.X's outputs and 5-9% of F^T.R's at M = 5003;
// groups of 128 or 64 leave fewer and were slower for their drains (solves of
// M = 10^4: 190 and 218 ms against 182).
//
// This replaces ~12 FP32 operations a term on the CUDA cores by 29 bf16 MMA
// terms.  One CTA per SM walks a list of 128 x BN output tiles.  The slices
// (digits and magnitudes) of a K chunk are one TMA box each: A 8 x 128 rows, B
// 8 x BN rows of 64 bytes (64-byte swizzle).  B's digits are stored even ones
// first (0 2 4 6 1 3 5) and so are the levels' accumulators, so with one digit
// of A the even digits of B are consecutive rows whose products belong to
// consecutive accumulators, and the odd ones too: 13 MMA instructions a K
// slice, N up to 256, instead of 28.  They alternate between the two halves of
// the accumulators, for an MMA starts late behind one that it shares columns
// with (with six digits, 21 pairs: without the alternation 9 instructions took
// 1350 cycles a K slice, with it 11 took 1150, for 672 of arithmetic).  BN =
// 64 fills the 512 tensor-memory columns; a stage is 96 KB and two fit.  The
// drain is not overlapped with the MMAs (no room for a second accumulator),
// eight warps share it; the output of a tile is formed, almost without the
// FP64 pipe, and stored while the next tile's MMAs run.
#pragma once

#include <algorithm>
#include <cmath>

#include "tc_band.cuh"

namespace pqdts {

constexpr int kDgDigits = 7;  // base-256 digits an operand
constexpr int kDgSlices = kDgDigits + 1;  // ... and its magnitudes
// Terms of at most 1/2 x 1/2 whose sums, in units of 2^-(48 + fine) of the
// scales, stay below 2^63 (fine = dg_fine(K) >= 0); F.X, which cancels with P,
// takes units of 2^-52 and finer only.
constexpr int kDgMaxFwd = 1 << 13, kDgMaxTrans = 1 << 17;
constexpr int kDgChunks = 8;   // K chunks (of kTcK) of a group
constexpr int kDgGroup = kDgChunks * kTcK;
constexpr int kDgThreads = 320;  // TMA warp, MMA warp, 8 epilogue warps
constexpr int kDgMaxStages = 4;
constexpr uint32_t kDgRing = 216u * 1024u;

// Place of B's digit q, and of level q's accumulator.
__host__ __device__ constexpr int dg_slot(int q) { return (q & 1) * ((kDgDigits + 1) / 2) + (q >> 1); }

// Bits below 2^-48 of the scales' product in which sums of at most `terms`
// terms are kept (at most 8: level 5 is then whole).
inline int dg_fine(int terms) {
  int fine = 8;
  while (fine > 0 && ((int64_t)terms << fine) >= kDgMaxTrans) --fine;
  return fine;
}

// The size, in units of the largest group's scales' product, that the sum of
// a digit product's |f| |x| must reach for its rounding (root mean squares:
// six dropped pairs of level 7 a term, digits of ~74 at a weight of 2^-72, and
// half a unit of the sum a drain) to stay below the double-FP32 kernels' (0.17
// sqrt(K) 2^-48 of the sum: on Poisson bands, K = 200 .. 1300, two such
// products leave 2.5 .. 6.5 * 2^-48 at the median entry of the gradient).
inline float dg_floor(int terms, int groups, int fine) {
  const double drop = std::sqrt((double)std::max(terms, 1)) * std::ldexp(1.0, -58);
  const double unit = std::sqrt((double)groups) * std::ldexp(0.29, -48 - fine);
  return (float)(std::hypot(drop, unit) / (std::sqrt((double)std::max(terms, 1)) * std::ldexp(0.17, -48)));
}

// Biased exponent of a double's magnitude (2047: infinite or NaN); of a scale:
// at least 1, 0 for no non-zero value.
__device__ __forceinline__ int dg_exponent(double v) { return (int)((__double_as_longlong(v) >> 52) & 0x7ff); }
__device__ __forceinline__ int dg_scale(double v) { return nonzero(v) ? max(1, dg_exponent(v)) : 0; }

// The S digits (bf16 bit patterns, most significant first) of v, whose biased
// exponent is at most emax >= 1 (or v = 0): v = 2^(emax - 1021 - 8 S) t, t =
// v's mantissa shifted to the scale's 8 S bits, rounded half away from zero;
// each byte of t + 0x8080...80 is a digit + 128.  Then |v| 2^(1021 - eall), below 1/2 (eall:
// the largest exponent of the whole row or column), truncated to bf16.
__device__ __forceinline__ void dg_digits(double v, int emax, int eall, uint32_t (&d)[kDgSlices]) {
  constexpr int S = kDgDigits;
  const long long b = __double_as_longlong(v);
  int e = (int)((b >> 52) & 0x7ff);
  unsigned long long m = (unsigned long long)b & ((1ull << 52) - 1);
  if (e != 0) m |= 1ull << 52;
  else e = 1;
  const int sh = emax - e + 54 - 8 * S;  // >= 54 - 8 S
  unsigned long long t;  // <= 2^(8 S - 1)
  if (sh <= 0) t = m << -sh;
  else t = sh <= 54 ? (m + (1ull << (sh - 1))) >> sh : 0ull;
  constexpr unsigned long long bias = 0x8080808080808080ull >> (64 - 8 * S);
  const unsigned long long u = (b < 0 ? 0ull - t : t) + bias;
#pragma unroll
  for (int q = 0; q < S; ++q) {
    const uint32_t byte = (uint32_t)(u >> (8 * (S - 1 - q))) & (q == 0 ? 0x1ffu : 0xffu);
    // 2^23 + byte as a float, minus 2^23 + 128: the digit, exactly
    d[q] = __float_as_uint(__fsub_rn(__uint_as_float(0x4b000000u | byte), 8388736.0f)) >> 16;
  }
  const int be = dg_exponent(v) - eall + 125;  // (subnormal: none)
  d[S] = be > 0 && dg_exponent(v) > 0 ? ((uint32_t)be << 7) | ((uint32_t)(b >> 45) & 0x7fu) : 0u;
}

// What a digit product takes from each column n of X (R x N row-major): its
// scale in each group g of rows, into exps[g N + n]; its scale over all rows,
// and its first and last non-zero row as R - first and last + 1 (0: none), into
// col[n], col[N + n] and col[2 N + n] (zeroed by the caller).  Block: 32
// columns x one group.
__global__ void __launch_bounds__(256) k_dg_columns(const double* __restrict__ X, int R, int N, int* __restrict__ col,
                                                    int* __restrict__ exps) {
  __shared__ int s[3][8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int n = blockIdx.x * 32 + lane, r0 = blockIdx.y * kDgGroup;
  int v[3] = {0, 0, 0};
  if (n < N)
#pragma unroll 4
    for (int r = r0 + w; r < min(R, r0 + kDgGroup); r += 8) {
      const double x = X[(int64_t)r * N + n];
      v[0] = max(v[0], dg_scale(x));
      if (nonzero(x)) {
        v[1] = max(v[1], R - r);
        v[2] = r + 1;
      }
    }
#pragma unroll
  for (int k = 0; k < 3; ++k) s[k][w][lane] = v[k];
  __syncthreads();
  if (w < 3 && n < N) {
    int m = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) m = max(m, s[w][q][lane]);
    if (w == 0) exps[(int64_t)blockIdx.y * N + n] = m;
    if (m > 0) atomicMax(col + w * N + n, m);
  }
}

// Digits of X (R x N row-major) as the products' K-major operand: digit q of
// X[r, n] at out[(dg_slot(q) * N + n) * ld + r] (ld >= R, even), its
// magnitude in slot S.  A block transposes 64 rows x 32 columns through shared
// memory; HBM bound (8 bytes in, 16 out).
__global__ void __launch_bounds__(256) k_dg_split_t(const double* __restrict__ X, int R, int N,
                                                    const int* __restrict__ col, const int* __restrict__ exps,
                                                    int64_t ld, uint16_t* __restrict__ out) {
  constexpr int S = kDgDigits;
  __shared__ __align__(4) uint16_t t[kDgSlices][32][66];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int r0 = blockIdx.x * 64, n0 = blockIdx.y * 32;
  {
    const int n = n0 + lane;
    const int emax = n < N ? exps[(int64_t)(r0 / kDgGroup) * N + n] : 0, eall = n < N ? col[n] : 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int y = w + 8 * k, r = r0 + y;
      const double v = (r < R && n < N) ? X[(int64_t)r * N + n] : 0.0;
      uint32_t d[kDgSlices];
      dg_digits(v, emax, eall, d);
#pragma unroll
      for (int q = 0; q <= S; ++q) t[q < S ? dg_slot(q) : S][lane][y] = (uint16_t)d[q];
    }
  }
  __syncthreads();
  const int r = r0 + 2 * lane;
#pragma unroll 4
  for (int x = w; x < kDgSlices * 32; x += 8) {
    const int q = x >> 5, n = n0 + (x & 31);
    if (n >= N || r >= R) continue;
    uint16_t* o = out + ((int64_t)q * N + n) * ld + r;
    if (r + 1 < R) *reinterpret_cast<uint32_t*>(o) = *reinterpret_cast<const uint32_t*>(&t[q][x & 31][2 * lane]);
    else *o = t[q][x & 31][2 * lane];
  }
}

// Band of row r of F (TRANS: F^T): first column, width, offset of its values.
template <bool TRANS>
__device__ __forceinline__ void dg_row(const DevBands& f, int r, int& lo, int& w, int64_t& off) {
  lo = w = 0;
  off = 0;
  if (TRANS) {
    off = f.tptr[r];
    w = (int)(f.tptr[r + 1] - off);
    if (w > 0) lo = f.tidx[off];
  } else if (f.flo[r] >= 0) {
    lo = f.flo[r];
    w = f.fw[r];
    off = f.foff[r];
  }
}

// Digits of the band operand: row r's values val[off .. off + w) at columns
// lo .. lo + w - 1 of F (TRANS: of F^T, whose rows are contiguous in d) ->
// digit q at out[(q * rows + r) * kmax + (column - kb[r / 128])], zero
// elsewhere, the magnitudes as digit S; the row's scale into rowall[r], and
// that in the j-th group from kb's on into rowexp[r * groups + j].  One block
// per padded row.
template <bool TRANS>
__global__ void __launch_bounds__(256) k_dg_band(DevBands f, const double* __restrict__ val,
                                                 const int32_t* __restrict__ kb, int rows, int kmax, int groups,
                                                 uint16_t* __restrict__ out, int* rowexp, int* __restrict__ rowall) {
  __shared__ int s_e;
  const int r = blockIdx.x, R = TRANS ? f.M : f.D, lane = threadIdx.x & 31;
  int lo = 0, w = 0;
  int64_t off = 0;
  if (r < R) dg_row<TRANS>(f, r, lo, w, off);
  if (threadIdx.x == 0) s_e = 0;
  __syncthreads();
  const int b0 = max(kb[r / kTcRows], 0), g0 = b0 / kDgGroup;
  int* exps = rowexp + (int64_t)r * groups;
  for (int j = threadIdx.x >> 5; j < groups; j += 8) {
    const int k0 = max((g0 + j) * kDgGroup - lo, 0), k1 = min((g0 + j + 1) * kDgGroup - lo, w);
    int e = 0;
    for (int k = k0 + lane; k < k1; k += 32) e = max(e, dg_scale(val[off + k]));
    e = __reduce_max_sync(0xffffffffu, (unsigned)e);
    if (lane == 0) {
      exps[j] = e;
      if (e > 0) atomicMax(&s_e, e);
    }
  }
  __syncthreads();
  const int eall = s_e;
  if (threadIdx.x == 0) rowall[r] = eall;
  const int start = lo - b0;  // first local column of the band
  for (int x = threadIdx.x; x < kmax; x += blockDim.x) {
    const int k = x - start;
    const double v = (unsigned)k < (unsigned)w ? val[off + k] : 0.0;
    uint32_t d[kDgSlices];
    dg_digits(v, exps[(b0 + x) / kDgGroup - g0], eall, d);
#pragma unroll
    for (int q = 0; q < kDgSlices; ++q) out[((int64_t)q * rows + r) * kmax + x] = (uint16_t)d[q];
  }
}

// 3-D TMA tile load (x, y, z = K, row, digit) completing on `bar`.
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// 8 consecutive columns of this thread's accumulator row, waited in place.
__device__ __forceinline__ void dg_ld8(uint32_t a, float (&v)[8]) {
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(a)
      : "memory");
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[j]);
}

// ... in each of the S levels (ls columns each).
__device__ __forceinline__ void dg_ld8_levels(uint32_t a, uint32_t ls, float (&v)[kDgDigits][8]) {
  uint32_t r[48];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%48];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%49];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%50];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%24, %25, %26, %27, %28, %29, %30, %31}, [%51];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%32, %33, %34, %35, %36, %37, %38, %39}, [%52];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%40, %41, %42, %43, %44, %45, %46, %47}, [%53];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]),
        "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]),
        "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47])
      : "r"(a + dg_slot(0) * ls), "r"(a + dg_slot(1) * ls), "r"(a + dg_slot(2) * ls), "r"(a + dg_slot(3) * ls),
        "r"(a + dg_slot(4) * ls), "r"(a + dg_slot(5) * ls)
      : "memory");
#pragma unroll
  for (int q = 0; q < 6; ++q)
#pragma unroll
    for (int j = 0; j < 8; ++j) v[q][j] = __uint_as_float(r[8 * q + j]);
  dg_ld8(a + dg_slot(6) * ls, v[6]);
}

// t * 2^e as a double, rounded to nearest (halves away from zero), by the
// integer pipes: the FP64 pipe takes 64 cycles an instruction, and a tile's
// outputs must be formed while the next tile's first MMAs run.
__device__ __forceinline__ double dg_value(long long t, int e) {
  const unsigned long long u = t < 0 ? 0ull - (unsigned long long)t : (unsigned long long)t;
  if (u == 0) return 0.0;
  const int lz = __clzll((long long)u), be = 1023 + 63 - lz + e;  // biased exponent
  if (be < 1 || be > 2046) return be < 1 ? 0.0 : (t < 0 ? -1.0 : 1.0) * __longlong_as_double(0x7ff0000000000000ll);
  const unsigned long long m = u << lz;  // leading one at bit 63
  const unsigned long long r = (m >> 11) + ((m >> 10) & 1);  // a carry raises the exponent
  return __longlong_as_double((long long)((((unsigned long long)(be - 1) << 52) + r) |
                                          ((unsigned long long)t & 0x8000000000000000ull)));
}

// acc 2^ea + s 2^es as an integer of 2^max(ea, es), rounded, and ea the larger.
__device__ __forceinline__ void dg_add(long long& acc, int& ea, long long s, int es) {
  const int d = es - ea, n = d < 0 ? -d : d;
  const long long big = d > 0 ? s : acc, small = d > 0 ? acc : s;
  acc = big + (n == 0 ? small : n > 62 ? 0 : ((small >> (n - 1)) + 1) >> 1);
  ea = max(ea, es);
}

// End of the group of a tile's K chunk c0, as a chunk of the tile (base: its
// first chunk's place in K).
__device__ __forceinline__ int dg_group_end(int c0, int base, int nk) {
  return min(nk, ((base + c0) / kDgChunks + 1) * kDgChunks - base);
}

// Operands and results of one digit product.
struct DgArgs {
  const int32_t *kb, *nch;           // K window of each 128-row block of A
  const int *rowexp, *rowall;        // scales of A's rows (k_dg_band) ...
  const int *colexp, *col;           // ... and of B's columns, over K rows (k_dg_columns)
  int K, groups, fine;
  const int32_t *sched_off, *sched_tile;  // each CTA's tiles (N tile fastest, then row block)
  int R, N, BN, stages;
  // what the epilogue adds (MODE 0, 3: P; MODE 4: the gamma stencil on V)
  const double* P;
  const double* V;
  double c2gam;
  double *out, *out2;
  // the outputs left to the double-FP32 kernels (DfRedo): those whose sum of
  // |a| |b| is below `floor` of the largest group's scales
  float floor;
  uint8_t* redo;
  int pitch;
  int* any;
  // F itself and B's FP64 values, for columns that hold an infinity or a NaN
  DevBands f;
  const double *val, *B;
  double* err;
  uint64_t wait_ns;
  int probe;
};

// Row r of F (TRANS: F^T) times column n of B in plain FP64: the result for
// a column with an infinite or NaN entry, which has no digits.
template <bool TRANS>
__device__ __noinline__ double dg_plain(const DgArgs& g, int r, int n) {
  int lo, w;
  int64_t off;
  dg_row<TRANS>(g.f, r, lo, w, off);
  double s = 0.0;
  for (int k = 0; k < w; ++k) s = fma(g.val[off + k], g.B[(int64_t)(lo + k) * g.N + n], s);
  return s;
}

// MODE 0: out = 2 (F.B - P); MODE 3: out = F.B - P (R = D rows of F);
// MODE 4: F^T.B + the gamma stencil on V into out and / or out2 (R = M rows
// of F^T; either may be null).  Every wait is bounded as in k_tc_band, with
// the same test hook; a wait that runs out sets *err and the CTA stores nothing
// more (the tiles before are stored, and other CTAs' may be: the result is
// undefined), lets the copies and MMAs in flight finish and frees its tensor
// memory.
template <int MODE>
__global__ void __launch_bounds__(kDgThreads, 1)
    k_dg_band_product(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB,
                      const __grid_constant__ DgArgs g) {
  constexpr int S = kDgDigits;
  extern __shared__ uint8_t tc_smem_raw[];
  __shared__ uint64_t bar_full[kDgMaxStages], bar_empty[kDgMaxStages], bar_accf, bar_acce, bar_fin, bar_probe;
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort;
  __shared__ int s_issued, s_consumed;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int BN = g.BN, N = g.N, stages = g.stages;
  const int ntn = (N + BN - 1) / BN;
  const uint32_t raw = smem_u32(tc_smem_raw);
  uint8_t* base = tc_smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  const uint32_t a_slice = kTcRows * kTcRowBytes, b_slice = (uint32_t)BN * kTcRowBytes;
  const uint32_t a_bytes = kDgSlices * a_slice, stage_bytes = a_bytes + kDgSlices * b_slice;
  const uint32_t ncols = kDgSlices * BN <= 128 ? 128u : kDgSlices * BN <= 256 ? 256u : 512u;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&mA);
    tma_prefetch_desc(&mB);
    for (int i = 0; i < stages; ++i) {
      mbar_init(&bar_full[i], 1);
      mbar_init(&bar_empty[i], 1);
    }
    mbar_init(&bar_accf, 1);
    mbar_init(&bar_acce, 256);
    mbar_init(&bar_fin, 1);
    mbar_init(&bar_probe, 1);
    s_abort = 0;
    s_issued = 0;
    s_consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    tc_alloc(&s_tmem, ncols);
    tc_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  const int j_begin = g.sched_off[blockIdx.x], j_end = g.sched_off[blockIdx.x + 1];

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      if (g.probe && !mbar_wait(&bar_probe, 0, g.wait_ns)) s_abort = 1;  // nothing arrives: runs out
      for (int j = j_begin; j < j_end && !s_abort; ++j) {
        const int t = g.sched_tile[j], nt = t % ntn, blk = t / ntn, kb = g.kb[blk];
        const int nk = kb >= 0 ? g.nch[blk] : 0;
        for (int ch = 0; ch < nk && !s_abort; ++ch, ++it) {
          const int st = it % stages;
          const uint32_t ph = (uint32_t)(it / stages) & 1u;
          if (!mbar_wait(&bar_empty[st], ph ^ 1u, g.wait_ns)) {
            s_abort = 1;
            break;
          }
          uint8_t* sa = base + (size_t)st * stage_bytes;
          mbar_expect_tx(&bar_full[st], stage_bytes);
          tma_load_3d(sa, &mA, ch * kTcK, blk * kTcRows, 0, &bar_full[st]);
          tma_load_3d(sa + a_bytes, &mB, kb + ch * kTcK, nt * BN, 0, &bar_full[st]);
          s_issued = it + 1;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int it = 0;
      uint32_t drain = 0;
      for (int j = j_begin; j < j_end && !s_abort; ++j) {
        const int blk = g.sched_tile[j] / ntn;
        const int kb = g.kb[blk], nk = kb >= 0 ? g.nch[blk] : 0;
        for (int c0 = 0, c1; c0 < nk && !s_abort; c0 = c1, ++drain) {
          if (!mbar_wait(&bar_acce, (drain & 1u) ^ 1u, g.wait_ns)) {  // accumulator drained
            s_abort = 1;
            break;
          }
          tc_fence_after();
          c1 = dg_group_end(c0, kb / kTcK, nk);
          for (int ch = c0; ch < c1; ++ch, ++it) {
            const int st = it % stages;
            const uint32_t ph = (uint32_t)(it / stages) & 1u;
            if (!mbar_wait(&bar_full[st], ph, g.wait_ns)) {
              s_abort = 1;
              break;
            }
            s_consumed = it + 1;
            tc_fence_after();
            const uint32_t sa = smem_u32(base + (size_t)st * stage_bytes), sb = sa + a_bytes;
#pragma unroll
            for (int k = 0; k < kTcK / 16; ++k) {
              const uint32_t o = 32u * k;
#pragma unroll
              for (int p = 0; p < S; ++p) {
                // A's digit p with B's even digits, then its odd ones (odd p:
                // the other way round, so that the halves of the accumulators
                // take turns), up to digit S - 1 - p.  The first products of a
                // drain overwrite the accumulators: digit 0 of A does that
                // for all levels.
                const uint32_t acc0 = (ch > c0 || k > 0 || p > 0) ? 1u : 0u;
                const uint64_t da = swz_desc(sa + (uint32_t)p * a_slice + o);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const int par = h ^ (p & 1), nq = (S - p - par + 1) / 2;
                  if (nq > 0)
                    tc_mma(tmem + (uint32_t)(dg_slot(p + par) * BN), da,
                           swz_desc(sb + (uint32_t)dg_slot(par) * b_slice + o), tc_idesc_bf16(kTcRows, nq * BN),
                           acc0);
                }
              }
              // the magnitudes, over all of the tile's K
              tc_mma(tmem + (uint32_t)(S * BN), swz_desc(sa + (uint32_t)S * a_slice + o),
                     swz_desc(sb + (uint32_t)S * b_slice + o), tc_idesc_bf16(kTcRows, BN), (ch > 0 || k > 0) ? 1u : 0u);
            }
            tc_commit(&bar_empty[st]);
          }
          tc_commit(&bar_accf);
        }
      }
      tc_commit(&bar_fin);  // arrives once every MMA this CTA issued is done (aborted or not)
    }
  } else {
    // epilogue: warp w reads tensor-memory lanes 32 (w % 4) .. + 31 (rows of
    // the tile), and one half of the N tile's columns
    const int q = warp & 3, half = (warp - 2) >> 2;
    const int hc = BN >> 1;  // columns per half: 8 .. 32
    const float low = __uint_as_float((uint32_t)(127 - 8 + g.fine) << 23);  // level 5 in units
    uint32_t drain = 0;
    bool ok = true;
    for (int j = j_begin; j < j_end && ok; ++j) {
      const int t = g.sched_tile[j], nt = t % ntn, blk = t / ntn;
      const int kb = g.kb[blk], nk = kb >= 0 ? g.nch[blk] : 0;
      const int rp = blk * kTcRows + q * 32 + lane;  // padded row
      // sums in units of 2^-fine of level 4's weight and their exponents (row
      // + column; 0: no group in which both have a value); what is below the
      // unit enters rounded to it
      long long acc[32];
      int ea[32];
      uint32_t left = 0;  // columns whose magnitudes' sum is below the floor
#pragma unroll
      for (int x = 0; x < 32; ++x) {
        acc[x] = 0;
        ea[x] = 0;
      }
      for (int c0 = 0, c1; c0 < nk; c0 = c1, ++drain) {
        c1 = dg_group_end(c0, kb / kTcK, nk);
        const int gk = (kb + c0 * kTcK) / kDgGroup;
        const int er = g.rowexp[(int64_t)rp * g.groups + (gk - kb / kDgGroup)];
        ok = mbar_wait(&bar_accf, drain & 1u, g.wait_ns);
        ok = __all_sync(0xffffffffu, ok && !s_abort);
        if (!ok) break;
        tc_fence_after();
        const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * hc);
#pragma unroll
        for (int x = 0; x < 32; x += 8)
          if (x < hc) {
            float v[S][8];
            dg_ld8_levels(ta + (uint32_t)x, (uint32_t)BN, v);
#pragma unroll
            for (int y = 0; y < 8; ++y) {
              long long s = __float2int_rn(v[4][y]);
              s += (long long)__float2int_rn(v[3][y]) << 8;
              s += (long long)__float2int_rn(v[2][y]) << 16;
              s += (long long)__float2int_rn(v[1][y]) << 24;
              s += (long long)__float2int_rn(v[0][y]) << 32;
              s = (s << g.fine) + __float2int_rn(low * fmaf(v[6][y], 0.00390625f, v[5][y]));
              const int n = nt * BN + half * hc + x + y;
              const int ec = n < N ? g.colexp[(int64_t)gk * N + n] : 0;
              if (er != 0 && ec != 0) dg_add(acc[x + y], ea[x + y], s, er + ec);
            }
            if (c1 == nk) {
              dg_ld8(ta + (uint32_t)(S * BN + x), v[0]);
              const int ra = g.rowall[rp];
#pragma unroll
              for (int y = 0; y < 8; ++y) {
                const int n = nt * BN + half * hc + x + y;
                const int d = ea[x + y] - ra - (n < N ? g.col[n] : 0);  // <= 0
                const float least = g.floor * __uint_as_float((uint32_t)(127 + max(d, -100)) << 23);
                if (ea[x + y] != 0 && !(v[0][y] >= least)) left |= 1u << (x + y);
              }
            }
          }
        tc_fence_before();
        mbar_arrive(&bar_acce);
      }
      if (!ok) {
        s_abort = 1;
        break;
      }
      const int r = rp;
      if (r >= g.R) continue;
      // value = acc * 2^(ea - 2090 - fine)
      const int e0 = -2090 - g.fine;
      int lo, w;
      int64_t off;
      dg_row<MODE == 4>(g.f, r, lo, w, off);
      const int n0 = nt * BN + half * hc;
      const int64_t o0 = (int64_t)r * N + n0;
      // pairs of columns by 16-byte accesses where rows keep the alignment
      const bool vec = (N & 1) == 0 && (n0 & 1) == 0;
      const double2 zero2 = make_double2(0.0, 0.0);
#pragma unroll
      for (int x = 0; x < 32; x += 2) {
        if (x >= hc || n0 + x >= N) continue;
        const bool two = n0 + x + 1 < N;
        const int64_t o = o0 + x;
        auto load = [&](const double* p) {
          if (vec) return *reinterpret_cast<const double2*>(p);
          return make_double2(p[0], two ? p[1] : 0.0);
        };
        auto store = [&](double* p, double2 y) {
          if (vec) {
            *reinterpret_cast<double2*>(p) = y;
          } else {
            p[0] = y.x;
            if (two) p[1] = y.y;
          }
        };
        const int* col = g.col + n0 + x;
        const int ce0 = col[0], ce1 = two ? col[1] : 0;
        // kept all the same: columns formed in FP64, and sums without a term
        // (the band ends before the column's first non-zero row, or begins
        // after its last)
        if (ce0 == 2047 || col[2 * N] <= lo || g.K - col[N] >= lo + w) left &= ~(1u << x);
        if (ce1 == 2047 || !two || col[2 * N + 1] <= lo || g.K - col[N + 1] >= lo + w) left &= ~(2u << x);
        double2 v = make_double2(dg_value(acc[x], ea[x] + e0), dg_value(acc[x + 1], ea[x + 1] + e0));
        if (ce0 == 2047) v.x = dg_plain<MODE == 4>(g, r, n0 + x);
        if (ce1 == 2047) v.y = dg_plain<MODE == 4>(g, r, n0 + x + 1);
        if (MODE != 4) {
          const double2 p = load(g.P + o);
          v.x -= p.x;
          v.y -= p.y;
          if (MODE == 0) v = make_double2(twice(v.x), twice(v.y));
          store(g.out + o, v);
        } else {
          if (g.c2gam != 0.0) {
            const double2 vi = load(g.V + o);
            const double2 vn = r < g.R - 1 ? load(g.V + o + N) : zero2, vp = r > 0 ? load(g.V + o - N) : zero2;
            if (r < g.R - 1) {
              v.x = fma(g.c2gam, vi.x - vn.x, v.x);
              v.y = fma(g.c2gam, vi.y - vn.y, v.y);
            }
            if (r > 0) {
              v.x = fma(-g.c2gam, vp.x - vi.x, v.x);
              v.y = fma(-g.c2gam, vp.y - vi.y, v.y);
            }
          }
          if (g.out) store(g.out + o, v);
          if (g.out2) store(g.out2 + o, v);
        }
      }
      uint8_t* bits = g.redo + (int64_t)r * g.pitch + (n0 >> 3);
      uint32_t some = 0;
#pragma unroll
      for (int x = 0; x < 32; x += 8)
        if (x < hc && n0 + x < N) {
          const uint32_t b = (left >> x) & 0xffu;
          bits[x >> 3] = (uint8_t)b;
          some |= b;
        }
      if (some) *g.any = 1;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (s_abort && threadIdx.x == 0) {
    *g.err = 1.0;
    for (int it = s_consumed; it < s_issued; ++it)
      if (!mbar_wait(&bar_full[it % stages], (uint32_t)(it / stages) & 1u, g.wait_ns)) break;
    mbar_wait(&bar_fin, 0, g.wait_ns);
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tc_dealloc(tmem, ncols);
  }
}

// The outputs that a digit product left (redo), in FP64: a block per row and 32
// columns, lane = column, the row's band in kDgRedoWarps shares of one warp each
// (a row at a time in one warp took twice as long, bound by its loads); out,
// out2, P, V and the modes as k_dg_band_product's.  For products so small that
// the double-FP32 kernels' launches (splitting the operand, masks, product) and
// latencies are what they cost.
constexpr int kDgRedoWarps = 4;
template <int MODE>
__global__ void __launch_bounds__(32 * kDgRedoWarps)
    k_dg_redo(DevBands f, const double* __restrict__ val, const double* __restrict__ B, const double* __restrict__ P,
              const double* __restrict__ V, double c2gam, double* out, double* out2, DfRedo redo) {
  if (*redo.any == 0) return;
  __shared__ double part[kDgRedoWarps][32];
  const int N = f.N, R = MODE == 4 ? f.M : f.D, ng = (N + 31) >> 5;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x / ng, n = (blockIdx.x % ng) * 32 + lane;
  const bool need = n < N && ((redo.bits[(int64_t)r * redo.pitch + (n >> 3)] >> (n & 7)) & 1);
  if (!__any_sync(0xffffffffu, need)) return;  // the same in every warp
  int lo, w;
  int64_t off;
  dg_row<MODE == 4>(f, r, lo, w, off);
  const int k0 = (int)((int64_t)w * warp / kDgRedoWarps), k1 = (int)((int64_t)w * (warp + 1) / kDgRedoWarps);
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  if (need) {
    const double* a = val + off;
    const double* b = B + (int64_t)lo * N + n;
    int k = k0;
    for (; k + 8 <= k1; k += 8) {
      double x[8], y[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        x[q] = a[k + q];
        y[q] = b[(int64_t)(k + q) * N];
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) s[q & 3] = fma(x[q], y[q], s[q & 3]);
    }
    for (; k < k1; ++k) s[0] = fma(a[k], b[(int64_t)k * N], s[0]);
  }
  part[warp][lane] = (s[0] + s[1]) + (s[2] + s[3]);
  __syncthreads();
  if (warp > 0 || !need) return;
  double v = part[0][lane];
#pragma unroll
  for (int q = 1; q < kDgRedoWarps; ++q) v += part[q][lane];
  const int64_t o = (int64_t)r * N + n;
  if (MODE != 4) {
    v -= P[o];
    out[o] = MODE == 0 ? 2.0 * v : v;
    return;
  }
  if (c2gam != 0.0) {
    const double vi = V[o];
    if (r < R - 1) v = fma(c2gam, vi - V[o + N], v);
    if (r > 0) v = fma(-c2gam, V[o - N] - vi, v);
  }
  if (out) out[o] = v;
  if (out2) out2[o] = v;
}

}  // namespace pqdts
