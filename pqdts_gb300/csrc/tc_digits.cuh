// Banded products of FP64 operands on the tensor cores, by exact integer
// digits: the mixed path's gradient F^T.R (dL, pqdts.f90:975-1032) and its
// FP64-accurate objective checks F.X - P (L, 917-973).
//
// Every operand row of F (or F^T) and every column of X (or R) is scaled by
// a power of two, so that its largest magnitude lies in [1/4, 1/2), rounded
// to 8 S bits and written as S signed digits in base 256, each exact in bf16:
//   x = 2^E (d_0 2^-8 + d_1 2^-16 + ... ),  |d_q| <= 128.
// A product is then a sum over digit pairs, and the pairs p + q = L of one
// level L share a weight 2^(-8 (L + 2)), so level L needs one integer sum
//   S_L = sum_k sum_{p + q = L} dF_p[k] dX_q[k]
// which the MMAs (bf16 in, FP32 accumulator in tensor memory) form exactly:
// a product of digits is at most 2^14, and the accumulators are drained into
// 64-bit integers every kDgDrain = 8 chunks of K = 32, so a pair's sum stays
// within 256 * 2^14 = 2^22 and the levels 0..3 within 2^24, the integers an
// FP32 accumulator holds; the next ones may pass that (by at most 1.75x,
// operands whose digits all have one sign) and then round by an ulp.  The
// levels 0 .. S - 1 are kept, S (S + 1) / 2 digit pairs: the error of a sum
// is ~sqrt(K) 2^(1 - 8 S) of (row scale x column scale).
//
// S = 6 for F^T.R.  S = 7 for F.X, whose difference from P cancels and leaves
// that error larger beside it: at iterates with most entries zero six digits
// left the gradient 1.0-1.7 times (M = 200-400), 0.7 (M = 900), 0.2 times (M =
// 4000-10^4, single entries up to 1.6 times) as far from 64-bit arithmetic as
// the double-FP32 kernels (k_fwd_df, k_trans_df) do, seven 0.07-0.4 times at
// M = 200-400 and 0.04-0.1 above (dense iterates: 0.04-0.25), for 2 % more
// time of F.X at M = 6000 and 11 % at M = 10^4.
//
// This replaces ~12 FP32 operations a term on the CUDA cores by 28 (F^T: 21)
// bf16 MMA terms.  One CTA per SM walks a list of 128 x BN output tiles.  The
// digits of a K chunk are one TMA box each: A S x 128 rows, B S x BN rows of
// 64 bytes (64-byte swizzle).  B's digits are stored even ones first (0 2 4 6
// 1 3 5) and so are the levels' accumulators, so with one digit of A the even
// digits of B are consecutive rows whose products belong to consecutive
// accumulators, and the odd ones too: 13 (11) MMA instructions a K slice, N up
// to 256 (192), instead of 28 (21).  They alternate between the two halves of
// the accumulators, for an MMA starts late behind one that it shares columns
// with (S = 6: without the alternation 9 instructions, N up to 256, took 1350
// cycles a K slice, now ~1150, for 672 of arithmetic).  BN = 64 fills 448
// (384) of the 512 tensor-memory columns; a stage is 84 (72) KB and two
// (three) fit.  The drain is not overlapped with the MMAs (no room for a
// second accumulator), eight warps share it; the output of a tile is formed,
// almost without the FP64 pipe, and stored while the next tile's MMAs run.
#pragma once

#include "tc_band.cuh"

namespace pqdts {

constexpr int kDgFwd = 7, kDgTrans = 6;  // base-256 digits an operand
// The sums, in units of 2^-52 (2^-48) of the scales, stay below 2^63 for so
// many terms of at most 1/2 x 1/2.
constexpr int kDgMaxFwd = 1 << 13, kDgMaxTrans = 1 << 17;
constexpr int kDgDrain = 8;   // K chunks (of kTcK) between drains
constexpr int kDgThreads = 320;  // TMA warp, MMA warp, 8 epilogue warps
constexpr int kDgMaxStages = 4;
constexpr uint32_t kDgRing = 216u * 1024u;

// Place of B's digit q, and of level q's accumulator, among S.
template <int S>
__host__ __device__ constexpr int dg_slot(int q) {
  return (q & 1) * ((S + 1) / 2) + (q >> 1);
}

// Biased exponent of a double's magnitude (2047: infinite or NaN).
__device__ __forceinline__ int dg_exponent(double v) { return (int)((__double_as_longlong(v) >> 52) & 0x7ff); }

// The S digits (bf16 bit patterns, most significant first) of v, whose biased
// exponent is at most emax: v = 2^(emax - 1021 - 8 S) t, t = v's mantissa
// shifted to the scale's 8 S bits, rounded half away from zero; each byte of
// t + 0x8080...80 is a digit + 128.
template <int S>
__device__ __forceinline__ void dg_digits(double v, int emax, uint32_t (&d)[S]) {
  const long long b = __double_as_longlong(v);
  int e = (int)((b >> 52) & 0x7ff);
  unsigned long long m = (unsigned long long)b & ((1ull << 52) - 1);
  if (e != 0) m |= 1ull << 52;
  else e = 1;
  const int sh = max(emax, 1) - e + 54 - 8 * S;  // >= 54 - 8 S
  unsigned long long t;  // <= 2^(8 S - 1)
  if (S == 7 && sh <= 0) t = m << -sh;
  else t = sh <= 54 ? (m + (1ull << (sh - 1))) >> sh : 0ull;
  constexpr unsigned long long bias = 0x8080808080808080ull >> (64 - 8 * S);
  const unsigned long long u = (b < 0 ? 0ull - t : t) + bias;
#pragma unroll
  for (int q = 0; q < S; ++q) {
    const uint32_t byte = (uint32_t)(u >> (8 * (S - 1 - q))) & (q == 0 ? 0x1ffu : 0xffu);
    // 2^23 + byte as a float, minus 2^23 + 128: the digit, exactly
    d[q] = __float_as_uint(__fsub_rn(__uint_as_float(0x4b000000u | byte), 8388736.0f)) >> 16;
  }
}

// Largest biased exponent of each column of X (R x N row-major) into
// colexp[n] (zeroed by the caller): block (32 columns) x (a share of the
// rows, grid.y shares).
__global__ void __launch_bounds__(256) k_dg_colexp(const double* __restrict__ X, int R, int N,
                                                   int* __restrict__ colexp) {
  __shared__ int s[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int n = blockIdx.x * 32 + lane;
  int e = 0;
  if (n < N)
    for (int r = blockIdx.y * 8 + w; r < R; r += gridDim.y * 8) e = max(e, dg_exponent(X[(int64_t)r * N + n]));
  s[w][lane] = e;
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int q = 1; q < 8; ++q) e = max(e, s[q][lane]);
    if (n < N && e > 0) atomicMax(colexp + n, e);
  }
}

// Digits of X (R x N row-major) as the products' K-major operand: digit q of
// X[r, n] at out[(dg_slot<S>(q) * N + n) * ld + r] (ld >= R, even).  A block transposes
// 64 rows x 32 columns through shared memory; HBM bound (8 bytes in, 12 out).
template <int S>
__global__ void __launch_bounds__(256) k_dg_split_t(const double* __restrict__ X, int R, int N,
                                                    const int* __restrict__ colexp, int64_t ld,
                                                    uint16_t* __restrict__ out) {
  __shared__ __align__(4) uint16_t t[S][32][66];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int r0 = blockIdx.x * 64, n0 = blockIdx.y * 32;
  {
    const int n = n0 + lane;
    const int emax = n < N ? colexp[n] : 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int y = w + 8 * k, r = r0 + y;
      const double v = (r < R && n < N) ? X[(int64_t)r * N + n] : 0.0;
      uint32_t d[S];
      dg_digits<S>(v, emax, d);
#pragma unroll
      for (int q = 0; q < S; ++q) t[dg_slot<S>(q)][lane][y] = (uint16_t)d[q];
    }
  }
  __syncthreads();
  const int r = r0 + 2 * lane;
#pragma unroll 4
  for (int x = w; x < S * 32; x += 8) {
    const int q = x >> 5, n = n0 + (x & 31);
    if (n >= N || r >= R) continue;
    uint16_t* o = out + ((int64_t)q * N + n) * ld + r;
    if (r + 1 < R) *reinterpret_cast<uint32_t*>(o) = *reinterpret_cast<const uint32_t*>(&t[q][x & 31][2 * lane]);
    else *o = t[q][x & 31][2 * lane];
  }
}

// Digits of the band operand: row r's values val[off .. off + w) at columns
// lo .. lo + w - 1 of F (TRANS: of F^T, whose rows are contiguous in d) ->
// digit q at out[(q * rows + r) * kmax + (column - kb[r / 128])], zero
// elsewhere, and the row's exponent.  One block per padded row.
template <bool TRANS>
__global__ void __launch_bounds__(256) k_dg_band(DevBands f, const double* __restrict__ val,
                                                 const int32_t* __restrict__ kb, int rows, int kmax,
                                                 uint16_t* __restrict__ out, int* __restrict__ rowexp) {
  constexpr int S = TRANS ? kDgTrans : kDgFwd;
  __shared__ int s_e;
  const int r = blockIdx.x, R = TRANS ? f.M : f.D;
  int lo = 0, w = 0;
  int64_t off = 0;
  if (r < R) {
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
  if (threadIdx.x == 0) s_e = 0;
  __syncthreads();
  int e = 0;
  for (int k = threadIdx.x; k < w; k += blockDim.x) e = max(e, dg_exponent(val[off + k]));
  if (e > 0) atomicMax(&s_e, e);
  __syncthreads();
  e = s_e;
  if (threadIdx.x == 0) rowexp[r] = e;
  const int start = lo - max(kb[r / kTcRows], 0);  // first local column of the band
  for (int x = threadIdx.x; x < kmax; x += blockDim.x) {
    const int k = x - start;
    const double v = (unsigned)k < (unsigned)w ? val[off + k] : 0.0;
    uint32_t d[S];
    dg_digits<S>(v, e, d);
#pragma unroll
    for (int q = 0; q < S; ++q) out[((int64_t)q * rows + r) * kmax + x] = (uint16_t)d[q];
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

// 8 consecutive columns of this thread's accumulator row in each of the S
// levels (ls columns each), waited in place.
template <int S>
__device__ __forceinline__ void dg_ld8(uint32_t a, uint32_t ls, float (&v)[S][8]) {
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
      : "r"(a + dg_slot<S>(0) * ls), "r"(a + dg_slot<S>(1) * ls), "r"(a + dg_slot<S>(2) * ls),
        "r"(a + dg_slot<S>(3) * ls), "r"(a + dg_slot<S>(4) * ls), "r"(a + dg_slot<S>(5) * ls)
      : "memory");
#pragma unroll
  for (int q = 0; q < 6; ++q)
#pragma unroll
    for (int j = 0; j < 8; ++j) v[q][j] = __uint_as_float(r[8 * q + j]);
  if constexpr (S == 7) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(a + dg_slot<S>(6) * ls)
        : "memory");
#pragma unroll
    for (int j = 0; j < 8; ++j) v[S - 1][j] = __uint_as_float(r[j]);
  }
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

// Operands and results of one digit product.
struct DgArgs {
  const int32_t *kb, *nch;           // K window of each 128-row block of A
  const int *rowexp, *colexp;        // exponents of A's rows and B's columns
  const int32_t *sched_off, *sched_tile;  // each CTA's tiles (N tile fastest, then row block)
  int R, N, BN, stages;
  // what the epilogue adds (MODE 0, 3: P; MODE 4: the gamma stencil on V)
  const double* P;
  const double* V;
  double c2gam;
  double *out, *out2;
  // F itself and B's FP64 values, for columns that hold an infinity or a NaN
  DevBands f;
  const double *val, *B;
  double* err;
  uint64_t wait_ns;
};

// Row r of F (TRANS: F^T) times column n of B in plain FP64: the result for
// a column with an infinite or NaN entry, which has no digits.
template <bool TRANS>
__device__ __noinline__ double dg_plain(const DgArgs& g, int r, int n) {
  int lo = -1, w = 0;
  int64_t off = 0;
  if (TRANS) {
    off = g.f.tptr[r];
    w = (int)(g.f.tptr[r + 1] - off);
    if (w > 0) lo = g.f.tidx[off];
  } else if (g.f.flo[r] >= 0) {
    lo = g.f.flo[r];
    w = g.f.fw[r];
    off = g.f.foff[r];
  }
  double s = 0.0;
  for (int k = 0; k < w; ++k) s = fma(g.val[off + k], g.B[(int64_t)(lo + k) * g.N + n], s);
  return s;
}

// MODE 0: out = 2 (F.B - P); MODE 3: out = F.B - P (R = D rows of F);
// MODE 4: F^T.B + the gamma stencil on V into out and / or out2 (R = M rows
// of F^T; either may be null).  Every wait is bounded as in k_tc_band; a
// wait that runs out sets *err and the CTA stores nothing more, lets the
// copies and MMAs in flight finish and frees its tensor memory.
template <int MODE>
__global__ void __launch_bounds__(kDgThreads, 1)
    k_dg_band_product(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB,
                      const __grid_constant__ DgArgs g) {
  constexpr int S = MODE == 4 ? kDgTrans : kDgFwd;
  extern __shared__ uint8_t tc_smem_raw[];
  __shared__ uint64_t bar_full[kDgMaxStages], bar_empty[kDgMaxStages], bar_accf, bar_acce, bar_fin;
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort;
  __shared__ int s_issued, s_consumed;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int BN = g.BN, N = g.N, stages = g.stages;
  const int ntn = (N + BN - 1) / BN;
  const uint32_t raw = smem_u32(tc_smem_raw);
  uint8_t* base = tc_smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  const uint32_t a_slice = kTcRows * kTcRowBytes, b_slice = (uint32_t)BN * kTcRowBytes;
  const uint32_t a_bytes = S * a_slice, stage_bytes = a_bytes + S * b_slice;
  const uint32_t ncols = S * BN <= 128 ? 128u : S * BN <= 256 ? 256u : 512u;

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
        const int nk = g.kb[blk] >= 0 ? g.nch[blk] : 0;
        for (int c0 = 0; c0 < nk && !s_abort; c0 += kDgDrain, ++drain) {
          if (!mbar_wait(&bar_acce, (drain & 1u) ^ 1u, g.wait_ns)) {  // accumulator drained
            s_abort = 1;
            break;
          }
          tc_fence_after();
          const int c1 = min(nk, c0 + kDgDrain);
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
                    tc_mma(tmem + (uint32_t)(dg_slot<S>(p + par) * BN), da,
                           swz_desc(sb + (uint32_t)dg_slot<S>(par) * b_slice + o), tc_idesc_bf16(kTcRows, nq * BN),
                           acc0);
                }
              }
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
    uint32_t drain = 0;
    bool ok = true;
    for (int j = j_begin; j < j_end && ok; ++j) {
      const int t = g.sched_tile[j], nt = t % ntn, blk = t / ntn;
      const int nk = g.kb[blk] >= 0 ? g.nch[blk] : 0;
      // sums in units of level 4's weight (S = 7: a sixteenth of it); the
      // levels below enter rounded to the unit
      constexpr int fine = S == 7 ? 4 : 0;
      long long acc[32];
#pragma unroll
      for (int x = 0; x < 32; ++x) acc[x] = 0;
      for (int c0 = 0; c0 < nk; c0 += kDgDrain, ++drain) {
        ok = mbar_wait(&bar_accf, drain & 1u, g.wait_ns);
        ok = __all_sync(0xffffffffu, ok && !s_abort);
        if (!ok) break;
        tc_fence_after();
        const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * hc);
#pragma unroll
        for (int x = 0; x < 32; x += 8)
          if (x < hc) {
            float v[S][8];
            dg_ld8<S>(ta + (uint32_t)x, (uint32_t)BN, v);
#pragma unroll
            for (int y = 0; y < 8; ++y) {
              long long s;
              if constexpr (S == 7)
                s = (long long)__float2int_rn(v[4][y]) * 16 + __float2int_rn(0.0625f * fmaf(v[6][y], 0.00390625f, v[5][y]));
              else
                s = __float2int_rn(fmaf(v[5][y], 0.00390625f, v[4][y]));
              s += (long long)__float2int_rn(v[3][y]) << (8 + fine);
              s += (long long)__float2int_rn(v[2][y]) << (16 + fine);
              s += (long long)__float2int_rn(v[1][y]) << (24 + fine);
              s += (long long)__float2int_rn(v[0][y]) << (32 + fine);
              acc[x + y] += s;
            }
          }
        tc_fence_before();
        mbar_arrive(&bar_acce);
      }
      if (!ok) {
        s_abort = 1;
        break;
      }
      const int r = blk * kTcRows + q * 32 + lane;
      if (r >= g.R) continue;
      // value = acc * 2^(rowexp + colexp - 2090 - fine)
      const int er = g.rowexp[r] - 2090 - fine;
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
        const int ce0 = g.colexp[n0 + x], ce1 = two ? g.colexp[n0 + x + 1] : 0;
        double2 v = make_double2(dg_value(acc[x], er + ce0), dg_value(acc[x + 1], er + ce1));
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

}  // namespace pqdts
