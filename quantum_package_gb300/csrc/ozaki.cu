// FP64-accurate tall-skinny Gram blocks X = A^T B on the tensor cores
// (tcgen05, sm_103a) by error-free splitting of the FP64 operands into BF16
// digit planes (the Ozaki scheme: K. Ozaki, T. Ogita, S. Oishi, S. M. Rump,
// "Error-free transformations of matrix multiplication by using fast routines
// of matrix multiplication and its applications", Numer. Algorithms 59 (2012)
// 95-118), with exact integer accumulation of the digit products and FP64
// combination of the per-CTA results.
//
// Splitting.  Column c of an operand gets the exponent E_c with |x| < 2^E_c
// for every element (k_col_maxexp).  An element is rounded to the 56-bit
// fixed-point integer F = round(|x| 2^(56 - E_c)) and written in balanced
// base 128, F = sum_p d_p 2^(49 - 7p) with d_1..d_7 in [-64, 63] and d_0 in
// [0, 128], every digit times the sign of x: integers exact in BF16.  The
// digits below the first are those of F + 64 (1 + 2^7 + ... + 2^42) less 64
// each, so they come out of independent shifts and masks, with no carry chain.
// Balanced digits make both the rounding and the dropped low-order products
// zero-mean, so they do not pile up in sums of squares (Gram diagonals).
//
// Products.  For digit planes p of A and q of B, tcgen05.mma (kind::f16,
// BF16 x BF16 -> FP32, M = 128 columns of A, N = 16 columns of B, K = rows)
// forms sum_r d_p(a_ri) d_q(b_rj) exactly: a product is at most 2^14 (both
// leading digits) or 2^13, and a level L = p + q over 128 rows stays below
// 2^23, so the FP32 accumulator of each level holds an exact integer.
// Levels L = 0..7 are kept (a dropped product is below 2^-56 of
// max|a| max|b|, like the rounding of the splitting).  Every 128 rows (a
// window) the eight level accumulators are read from tensor memory and added,
// as integers, to two int64 fixed-point sums per entry (levels 0-3 and 4-7),
// so nothing is rounded until the CTA's rows are done; then each CTA's entry
// becomes an FP64 value and the CTAs are summed in FP64 in a fixed order.
//
// Pipeline (one CTA per SM over a contiguous block of rows, chunks of 32
// rows), one role per warp:
//  * the last warp streams the raw FP64 rows of each chunk into a ring of raw
//    stages (cp.async.bulk per operand block, completing on rawfull[r]; a
//    block whose rows are strided or unaligned is copied by the warp's lanes);
//  * warps 0-11 (those that have tasks) cut the chunk into digit planes (stores of
//    2, 4 or 8 rows of one column), free the raw stage (rawempty[r]) and fill digit stage s
//    (full[s]);
//  * one warp issues the chunk's 16 MMAs once full[s] completes and commits
//    them to empty[s] and, at the end of a window, to accf[b]; the windows
//    rotate over four tensor-memory accumulator buffers b;
//  * four warps, whose lane quarters cover the 128 accumulator rows, add a
//    finished window to their int64 sums and arrive on acce[b], so that the
//    integer work never holds up the splitting.
// A plane p of A meets B planes 0..7-p only (levels p..7), so its MMA has
// N = (8 - p) 16 and writes the accumulator from level p on.
// Every mbarrier wait is bounded and gives up early once another warp has set
// the CTA's error flag; the warps then leave their loops, the kernel waits
// (bounded) for its bulk copies and MMAs, frees its tensor memory and sets
// *status.
#include <algorithm>

#include "block_ring.h"
#include "qpgpu_internal.cuh"

namespace {

constexpr int OZ_SPLIT = 384;                // splitting threads (warps 0-11)
constexpr int OZ_FLUSH_WARP = OZ_SPLIT / 32;       // the next 4 warps flush the accumulators (a multiple of 4)
constexpr int OZ_MMA_WARP = OZ_FLUSH_WARP + 4;     // issues the MMAs, owns the tensor memory
constexpr int OZ_LOAD_WARP = OZ_MMA_WARP + 1;      // streams the raw rows
constexpr int OZ_THREADS = (OZ_LOAD_WARP + 1) * 32;
static_assert(OZ_FLUSH_WARP % 4 == 0, "flush warp w reads the accumulator lanes of quarter w % 4");
constexpr int OZ_M = 128;                    // MMA M: columns of A (padded)
constexpr int OZ_N = 16;                     // columns of B (padded)
constexpr int OZ_KC = 32;                    // rows per chunk (MMA K = 2 x 16)
constexpr int OZ_DIG = 8;                    // digit planes per operand
constexpr int OZ_LEVELS = 8;                 // levels p + q = 0..7 kept
constexpr int OZ_WINDOW = 4;                 // chunks per accumulator window (128 rows)
constexpr int OZ_NBUF = 4;                   // accumulator buffers
constexpr int OZ_B_TILE = OZ_N * OZ_KC * 2;  // bytes of one B digit plane
constexpr int OZ_MAXST = 3;                  // digit stages at most
constexpr int OZ_TAB = 6144;  // alignment, exponents, block tables, barriers
constexpr int OZ_SMEM_MAX = 232448;
constexpr int OZ_MAXRAW = 8;  // raw stages at most
constexpr int OZ_MAXBLK = OZ_M + 2;  // operand blocks: at most one per column of A, two of B

constexpr int OZ_ACC_COLS = OZ_LEVELS * OZ_N;     // 128 tensor-memory columns per buffer
constexpr int OZ_TMEM_COLS = OZ_NBUF * OZ_ACC_COLS;  // 512: the whole tensor memory of the SM
constexpr long long OZ_WAIT_LIMIT = 1LL << 25;

// barrier slots
constexpr int OZ_B_FULL = 0, OZ_B_EMPTY = OZ_MAXST, OZ_B_ACCF = 2 * OZ_MAXST, OZ_B_ACCE = OZ_B_ACCF + OZ_NBUF,
              OZ_B_RAWF = OZ_B_ACCE + OZ_NBUF, OZ_B_RAWE = OZ_B_RAWF + OZ_MAXRAW, OZ_NBARS = OZ_B_RAWE + OZ_MAXRAW;

struct OzArgs {
  const double* A;  // blocks of nsdA columns, rows ldA values apart, blocks sA apart
  int64_t sA;
  int m, nsdA, ldA;
  const double* B0;  // nsdB columns, rows ldB apart
  const double* B1;  // optional second block (columns nsdB..2 nsdB-1)
  int nbc, nsdB, ldB;
  int64_t N, rows_per_cta;
  const int* eA;  // biased max exponent of each column of A (k_col_maxexp)
  const int* eB;
  double* partial;  // [cta][m][nbc]
  const int* skip;
  int* status;
  // digit stages: the 8 A planes (a_tile bytes each, the columns of A rounded
  // up to 8), then the 8 B planes, so that B planes 0..n-1 form one K-major
  // operand of 16 n rows.  An MMA reads 128 rows from each A plane: those past
  // its own are other digits, and their accumulator rows are never read.
  int nst, a_tile, stage;
  int nraw;        // raw stages in the ring
  int raw_stride;  // doubles per raw stage
  int rpt;         // rows per splitting task: 2, 4 or 8
  int nsw;         // splitting warps that have tasks
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// byte offset of element (row, k) in a K-major tile of 8 x 16-byte core
// matrices, core (row / 8, k / 8) at ((row / 8) * (KC / 8) + k / 8) * 128:
// the start of K step t is + t * 256, the K-direction stride (LBO) 128 bytes,
// the row-group stride (SBO) (KC / 8) * 128 = 512 bytes
__device__ __forceinline__ int kmaj(int row, int k) {
  return (((row >> 3) * (OZ_KC / 8)) + (k >> 3)) * 128 + (row & 7) * 16 + (k & 7) * 2;
}

// tcgen05 shared-memory matrix descriptor: start, LBO, SBO (bytes >> 4),
// descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t sdesc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(512 >> 4) << 32) |
         ((uint64_t)1 << 46);
}

// instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N >> 3 at bit 17, M >> 4 at bit 24
__device__ __forceinline__ uint32_t oz_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(OZ_M >> 4) << 24);
}

// 64 in every base-128 digit position of a 56-bit integer but the first
constexpr unsigned long long OZ_H = 64ull * ((1ull << 42) | (1ull << 35) | (1ull << 28) | (1ull << 21) |
                                             (1ull << 14) | (1ull << 7) | 1ull);

// 2 (F + OZ_H) + (0 or 1) of x against the biased max exponent eb
// (|x| < 2^(eb - 1022)): F = round(|x| 2^(56 - E)), E = eb - 1022, is the
// 53-bit significand times 2^3 shifted right by eb - ex and rounded (half
// up).  Shifted one bit less, the rounding is the carry of an added 1, and it
// and the digit offsets are one addition; the digits then sit one bit higher.
__device__ __forceinline__ unsigned long long oz_fixed(uint32_t bh, uint32_t bl, int eb) {
  const int ex = (int)((bh >> 20) & 0x7FF);
  int k = min(max(eb - ex, 0), 63);
  if (ex == 0) k = 63;  // zeros and subnormals: F = 0
  const uint32_t mh = __funnelshift_l(bl, (bh & 0xFFFFFu) | 0x100000u, 4), ml = bl << 4;
  return ((((unsigned long long)mh << 32) | ml) >> k) + (2 * OZ_H + 1);
}

// the 8 balanced digits of two values against the biased max exponents e0,
// e1, as BF16 pairs (x0 in the low half).  With G = F + OZ_H, the plain
// base-128 digits g_p of G give F = sum_p d_p 2^(49 - 7p) with d_0 = g_0 in
// [0, 128] and d_p = g_p - 64 in [-64, 63].  A digit n in the low bits of
// 0x4300 is the BF16 value 128 + n (128 gives 256), so a plane of both values
// is a mask and the exponent bits in one instruction and one packed FMA that
// takes off 128 (+ 64) and applies the signs, all exact; a pair of digits
// shares one 16-bit window of each value.  About 29 integer instructions a
// value, against about 40 with a digit at a time through FP32.
__device__ __forceinline__ uint32_t bf16_fma2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ void oz_digits2(double x0, double x1, int e0, int e1, uint32_t (&d)[OZ_DIG]) {
  const uint32_t h0 = (uint32_t)__double2hiint(x0), l0 = (uint32_t)__double2loint(x0);
  const uint32_t h1 = (uint32_t)__double2hiint(x1), l1 = (uint32_t)__double2loint(x1);
  const unsigned long long g0 = oz_fixed(h0, l0, e0), g1 = oz_fixed(h1, l1, e1);
  const uint32_t a0 = (uint32_t)g0, b0 = (uint32_t)(g0 >> 32), a1 = (uint32_t)g1, b1 = (uint32_t)(g1 >> 32);
  // 16-bit windows of both values: digit pairs (6, 7) one bit up, (4, 5), (2, 3), (0, 1)
  const uint32_t w3 = __byte_perm(a0, a1, 0x5410), w2 = __byte_perm(a0 >> 15, a1 >> 15, 0x5410);
  const uint32_t w1 = __byte_perm(__funnelshift_r(a0, b0, 29), __funnelshift_r(a1, b1, 29), 0x5410);
  const uint32_t w0 = __byte_perm(b0 >> 11, b1 >> 11, 0x5410);
  const uint32_t sg = __byte_perm(h0, h1, 0x7632) & 0x80008000u;
  const uint32_t one = sg | 0x3F803F80u, c128 = sg ^ 0xC300C300u, c192 = sg ^ 0xC340C340u;  // +-1, -+128, -+192
  d[0] = bf16_fma2(((w0 >> 7) & 0x00FF00FFu) | 0x43004300u, one, c128);
  d[1] = bf16_fma2((w0 & 0x007F007Fu) | 0x43004300u, one, c192);
  d[2] = bf16_fma2(((w1 >> 7) & 0x007F007Fu) | 0x43004300u, one, c192);
  d[3] = bf16_fma2((w1 & 0x007F007Fu) | 0x43004300u, one, c192);
  d[4] = bf16_fma2(((w2 >> 7) & 0x007F007Fu) | 0x43004300u, one, c192);
  d[5] = bf16_fma2((w2 & 0x007F007Fu) | 0x43004300u, one, c192);
  d[6] = bf16_fma2(((w3 >> 8) & 0x007F007Fu) | 0x43004300u, one, c192);
  d[7] = bf16_fma2(((w3 >> 1) & 0x007F007Fu) | 0x43004300u, one, c192);
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

// bounded wait for the completion of phase `parity` of an mbarrier; gives up
// early once the CTA's error flag is set
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const int* sflag) {
  for (long long it = 0; it < OZ_WAIT_LIMIT; ++it) {
    if (mbar_try(bar, parity)) return true;
    if ((it & 255) == 255 && *(volatile const int*)sflag) return false;
  }
  return false;
}

// bounded wait that ignores the error flag: for the drains before exit
__device__ __forceinline__ bool mbar_drain(uint32_t bar, uint32_t parity) {
  for (long long it = 0; it < OZ_WAIT_LIMIT; ++it)
    if (mbar_try(bar, parity)) return true;
  return false;
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// i 2^k exactly, |i| < 2^51, -1022 <= k <= 960: i is added to the low bits of
// 1.5 2^52, and one FMA scales it and takes the offset off.  (The 64-bit
// conversion instructions run on the FP64 pipe, two lanes a clock, several
// times each.)
__device__ __forceinline__ double scaled_int(long long i, int k) {
  const double x = __longlong_as_double(i + 0x4338000000000000ll);
  const double s = __longlong_as_double((long long)(k + 1023) << 52);
  const double off = __longlong_as_double(((long long)(k + 1023 + 52) << 52) | 0x8008000000000000ll);  // -1.5 2^(52 + k)
  return __fma_rn(x, s, off);
}

// level L of accumulator buffer `buf` (this warp's 32 lanes, 16 columns),
// exact integers below 2^23, shifted by sh into acc
__device__ __forceinline__ void oz_flush1(uint32_t taddr, int sh, long long (&acc)[OZ_N]) {
  uint32_t v[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < OZ_N; ++j) acc[j] += (long long)__float2int_rn(__uint_as_float(v[j])) << sh;
}

// RPT rows of one column (rows wcol doubles apart, nr of them real) into each
// of the 8 planes, `tile` bytes apart
template <int RPT>
__device__ __forceinline__ void oz_split_task(const double* xs, int wcol, int nr, int eb, uint8_t* dst, int tile) {
  uint32_t pk[OZ_DIG][RPT / 2];
#pragma unroll
  for (int k = 0; k < RPT; k += 2) {
    uint32_t d[OZ_DIG];
    oz_digits2(k < nr ? xs[k * wcol] : 0.0, k + 1 < nr ? xs[(k + 1) * wcol] : 0.0, eb, eb, d);
#pragma unroll
    for (int p = 0; p < OZ_DIG; ++p) pk[p][k >> 1] = d[p];
  }
#pragma unroll
  for (int p = 0; p < OZ_DIG; ++p) {
    if constexpr (RPT == 8)
      *reinterpret_cast<uint4*>(dst + p * tile) = make_uint4(pk[p][0], pk[p][1], pk[p][2], pk[p][3]);
    else if constexpr (RPT == 4)
      *reinterpret_cast<uint2*>(dst + p * tile) = make_uint2(pk[p][0], pk[p][1]);
    else
      *reinterpret_cast<uint32_t*>(dst + p * tile) = pk[p][0];
  }
}

template <int RPT>
__device__ __forceinline__ void oz_split(const double* rsrc, uint8_t* sa, uint8_t* sb, int m, int rw, int nrow,
                                         const int* coff, const int* cw, const int* sE, int tid, int a_tile) {
  const int ntask = rw * (OZ_KC / RPT);
  for (int t = tid; t < ntask; t += OZ_SPLIT) {
    const int grp = t / rw, col = t - grp * rw;
    const bool isA = col < m;
    const int cc = isA ? col : col - m;
    const int eb = sE[isA ? cc : OZ_M + cc];
    const int wcol = cw[col], k0 = RPT * grp;
    oz_split_task<RPT>(rsrc + coff[col] + k0 * wcol, wcol, nrow - k0, eb, (isA ? sa : sb) + kmaj(cc, k0),
                       isA ? a_tile : OZ_B_TILE);
  }
}

__global__ void __launch_bounds__(OZ_THREADS, 1) k_gram_oz(OzArgs g) {
  if (g.skip && *g.skip) return;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sbase = (uint8_t*)(((uintptr_t)smem + 1023) & ~(uintptr_t)1023);
  uint8_t* tiles = sbase;                                 // digit stage s: A planes, then B planes
  const int nst = g.nst;
  double* raw = (double*)(sbase + nst * g.stage);         // nraw stages, operand blocks of [OZ_KC][width]
  const double** bsrc = (const double**)(raw + (size_t)g.nraw * g.raw_stride);  // block bases
  int* bw = (int*)(bsrc + OZ_MAXBLK);                     // [OZ_MAXBLK] block widths
  int* bld = bw + OZ_MAXBLK;                              // [OZ_MAXBLK] row strides
  int* boff = bld + OZ_MAXBLK;                            // [OZ_MAXBLK] raw-stage offsets (doubles)
  int* coff = boff + OZ_MAXBLK;                           // [OZ_M + OZ_N] raw offset of each column
  int* cw = coff + OZ_M + OZ_N;                           // [OZ_M + OZ_N] width of its block
  int* sE = cw + OZ_M + OZ_N;                             // [OZ_M] A, [OZ_N] B exponents
  uint64_t* bars = (uint64_t*)(((uintptr_t)(sE + OZ_M + OZ_N) + 7) & ~(uintptr_t)7);
  uint32_t* tmem_slot = (uint32_t*)(bars + OZ_NBARS);
  int* sflag = (int*)(tmem_slot + 1);                     // error flag of the CTA
  int* snblk = sflag + 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m = g.m, nbc = g.nbc, rw = m + nbc;
  const uint32_t bar0 = smem_u32(bars);
  auto BAR = [&](int slot, int i) { return bar0 + 8u * (uint32_t)(slot + i); };

  for (int i = tid; i < nst * g.stage / 16; i += OZ_THREADS) reinterpret_cast<uint4*>(tiles)[i] = make_uint4(0, 0, 0, 0);
  for (int i = tid; i < OZ_M; i += OZ_THREADS) sE[i] = i < m ? g.eA[i] : 0;
  for (int j = tid; j < OZ_N; j += OZ_THREADS) sE[OZ_M + j] = j < nbc ? g.eB[j] : 0;
  if (warp == OZ_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(OZ_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int s = 0; s < OZ_MAXST; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(BAR(OZ_B_FULL, s)), "r"(g.nsw));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(BAR(OZ_B_EMPTY, s)));
    }
    for (int b = 0; b < OZ_NBUF; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(BAR(OZ_B_ACCF, b)));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(BAR(OZ_B_ACCE, b)));
    }
    for (int r = 0; r < OZ_MAXRAW; ++r) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(BAR(OZ_B_RAWF, r)));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(BAR(OZ_B_RAWE, r)), "r"(g.nsw));
    }
    asm volatile("fence.mbarrier_init.release.cluster;");
    *sflag = 0;
    // operand blocks: A in blocks of nsdA columns, then B0 and B1; each is
    // staged as [OZ_KC][width] at boff, its column c at coff[c] + row * width
    int nb = 0, col = 0, off = 0;
    for (int c0 = 0; c0 < m; c0 += g.nsdA, ++nb) {
      const int w = min(g.nsdA, m - c0);
      bsrc[nb] = g.A + (int64_t)(c0 / g.nsdA) * g.sA;
      bw[nb] = w;
      bld[nb] = g.ldA;
      boff[nb] = off;
      for (int j = 0; j < w; ++j, ++col) {
        coff[col] = off + j;
        cw[col] = w;
      }
      off += OZ_KC * w;
    }
    for (int c0 = 0; c0 < nbc; c0 += g.nsdB, ++nb) {
      const int w = min(g.nsdB, nbc - c0);
      bsrc[nb] = c0 == 0 ? g.B0 : g.B1;
      bw[nb] = w;
      bld[nb] = g.ldB;
      boff[nb] = off;
      for (int j = 0; j < w; ++j, ++col) {
        coff[col] = off + j;
        cw[col] = w;
      }
      off += OZ_KC * w;
    }
    *snblk = nb;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;

  const int64_t r0 = (int64_t)blockIdx.x * g.rows_per_cta;
  const int64_t r1 = min(r0 + g.rows_per_cta, g.N);
  const int nchunks = r1 > r0 ? (int)((r1 - r0 + OZ_KC - 1) / OZ_KC) : 0;
  const int nwin = (nchunks + OZ_WINDOW - 1) / OZ_WINDOW;
  const int nraw = g.nraw;

  if (warp < OZ_SPLIT / 32) {
    // ---- splitting warps -------------------------------------------------
    // up to 96 columns in tasks of 8 rows: a thread has the same task in every chunk
    const int ntask = rw * (OZ_KC / 8);
    const bool one = g.rpt == 8 && ntask <= OZ_SPLIT;
    int t_src = 0, t_w = 0, t_k0 = 0, t_e = 0, t_dst = 0, t_tile = 0;
    if (one && tid < ntask) {
      const int grp = tid / rw, col = tid - grp * rw;
      const bool isA = col < m;
      const int cc = isA ? col : col - m;
      t_k0 = 8 * grp;
      t_w = cw[col];
      t_src = coff[col] + t_k0 * t_w;
      t_e = sE[isA ? cc : OZ_M + cc];
      t_dst = (isA ? 0 : OZ_DIG * g.a_tile) + kmaj(cc, t_k0);
      t_tile = isA ? g.a_tile : OZ_B_TILE;
    }
    // digit stage s and raw stage rs of the chunk, and the parities of their uses
    int s = 0, rs = 0;
    uint32_t sp = 0, rp = 0;
    for (int c = 0; c < nchunks && warp < g.nsw; ++c) {
      // chunk c's raw rows have landed; the MMAs of chunk c - nst are done with digit stage s
      bool ok = mbar_wait(BAR(OZ_B_RAWF, rs), rp, sflag);
      if (ok && c >= nst) ok = mbar_wait(BAR(OZ_B_EMPTY, s), sp ^ 1u, sflag);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) atomicExch(sflag, 1);
        break;
      }
      uint8_t* sa = tiles + s * g.stage;
      uint8_t* sb = sa + OZ_DIG * g.a_tile;
      const double* rsrc = raw + (size_t)rs * g.raw_stride;
      const int nrow = (int)min((int64_t)OZ_KC, r1 - (r0 + (int64_t)c * OZ_KC));
      if (one) {
        if (tid < ntask) oz_split_task<8>(rsrc + t_src, t_w, nrow - t_k0, t_e, sa + t_dst, t_tile);
      } else if (g.rpt == 8)
        oz_split<8>(rsrc, sa, sb, m, rw, nrow, coff, cw, sE, tid, g.a_tile);
      else if (g.rpt == 4)
        oz_split<4>(rsrc, sa, sb, m, rw, nrow, coff, cw, sE, tid, g.a_tile);
      else
        oz_split<2>(rsrc, sa, sb, m, rw, nrow, coff, cw, sE, tid, g.a_tile);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(BAR(OZ_B_RAWE, rs));
        mbar_arrive(BAR(OZ_B_FULL, s));
      }
      if (++s == nst) s = 0, sp ^= 1u;
      if (++rs == nraw) rs = 0, rp ^= 1u;
    }
  } else if (warp < OZ_MMA_WARP) {
    // ---- flush warps: lane quarter q = warp % 4 holds rows 32 q .. 32 q + 31
    // (the sums live in this branch alone: the splitting warps need the registers)
    long long hi[OZ_N], lo[OZ_N];  // fixed-point sums of this thread's A column
#pragma unroll
    for (int j = 0; j < OZ_N; ++j) hi[j] = lo[j] = 0;
    const uint32_t lrow = (uint32_t)((warp & 3) * 32) << 16;
    for (int w = 0; w < nwin; ++w) {
      const int buf = w % OZ_NBUF;
      const bool ok = mbar_wait(BAR(OZ_B_ACCF, buf), (uint32_t)(w / OZ_NBUF) & 1u, sflag);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) atomicExch(sflag, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t ta = tmem + lrow + (uint32_t)(buf * OZ_ACC_COLS);
#pragma unroll
      for (int L = 0; L < OZ_LEVELS / 2; ++L) oz_flush1(ta + L * OZ_N, 7 * (3 - L), hi);
#pragma unroll
      for (int L = OZ_LEVELS / 2; L < OZ_LEVELS; ++L) oz_flush1(ta + L * OZ_N, 7 * (7 - L), lo);
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR(OZ_B_ACCE, buf));
    }
    const bool ok = *(volatile int*)sflag == 0;  // an error sets *status, whatever is written here
    const int i = (warp & 3) * 32 + lane;
    if (i < m)
#pragma unroll
      for (int j = 0; j < OZ_N; ++j)
        if (j < nbc) {
          const int e = (sE[i] - 1022) + (sE[OZ_M + j] - 1022);
          const double v = ldexp((double)hi[j], e - 35) + ldexp((double)lo[j], e - 63);
          g.partial[((int64_t)blockIdx.x * m + i) * nbc + j] = ok ? v : 0.0;
        }
  } else if (warp == OZ_MMA_WARP) {
    // ---- MMA warp: lane 0 issues, the warp stays converged ----------------
    uint32_t last_bar = 0, last_par = 0;  // the latest commit: its completion covers every MMA
    int s = 0;
    uint32_t sp = 0;
    for (int c = 0; c < nchunks; ++c) {
      const int w = c / OZ_WINDOW, buf = w % OZ_NBUF;
      bool ok = true;
      if (lane == 0) {
        // accumulator buffer flushed (window w - 4), digit stage s full
        if (c % OZ_WINDOW == 0 && w >= OZ_NBUF)
          ok = mbar_wait(BAR(OZ_B_ACCE, buf), (uint32_t)(w / OZ_NBUF - 1) & 1u, sflag);
        if (ok) ok = mbar_wait(BAR(OZ_B_FULL, s), sp, sflag);
        if (ok) {
          asm volatile("tcgen05.fence::after_thread_sync;");
          const bool first = (c % OZ_WINDOW) == 0;
          const uint32_t a0 = smem_u32(tiles + s * g.stage);
          const uint32_t b0 = a0 + OZ_DIG * g.a_tile;  // B planes 0..7
#pragma unroll
          for (int p = 0; p < OZ_DIG; ++p)
#pragma unroll
            for (int kt = 0; kt < OZ_KC / 16; ++kt) {
              // levels L = p..7 of A plane p against B planes 0..7-p; the
              // first product of a window overwrites the accumulator
              const uint32_t acc = (first && p == 0 && kt == 0) ? 0u : 1u;
              asm volatile(
                  "{\n .reg .pred pa;\n setp.ne.b32 pa, %4, 0;\n"
                  " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, pa;\n}" ::"r"(
                      tmem + (uint32_t)(buf * OZ_ACC_COLS + p * OZ_N)),
                  "l"(sdesc(a0 + p * g.a_tile + kt * 256)), "l"(sdesc(b0 + kt * 256)),
                  "r"(oz_idesc((OZ_LEVELS - p) * OZ_N)), "r"(acc));
            }
          mma_commit(BAR(OZ_B_EMPTY, s));
          last_bar = BAR(OZ_B_EMPTY, s);
          last_par = sp;
          if (c % OZ_WINDOW == OZ_WINDOW - 1 || c == nchunks - 1) mma_commit(BAR(OZ_B_ACCF, buf));
        } else {
          atomicExch(sflag, 1);
        }
      }
      if (!__shfl_sync(0xffffffffu, (int)ok, 0)) break;
      if (++s == nst) s = 0, sp ^= 1u;
    }
    // before the tensor memory is freed, every MMA issued must have completed
    if (lane == 0 && last_bar != 0 && !mbar_drain(last_bar, last_par)) atomicExch(sflag, 1);
    __syncwarp();
  } else if (warp == OZ_LOAD_WARP) {
    // ---- load warp: raw rows of chunk cc into raw stage cc % nraw ---------
    // A block whose rows are contiguous (row stride = width) and 16-byte
    // aligned comes in with one bulk copy; any other block is copied by the
    // lanes.  Rows past r1 are not copied: the split reads them as zeros.
    const int nblk = *snblk;
    int issued = 0;
    for (int cc = 0; cc < nchunks; ++cc) {
      const int rs = cc % nraw;
      const bool ok = cc < nraw || mbar_wait(BAR(OZ_B_RAWE, rs), (uint32_t)(cc / nraw - 1) & 1u, sflag);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) atomicExch(sflag, 1);
        break;
      }
      double* dst0 = raw + (size_t)rs * g.raw_stride;
      const int64_t rb = r0 + (int64_t)cc * OZ_KC;
      const int nrow = (int)min((int64_t)OZ_KC, r1 - rb);
      uint32_t bytes = 0;
      for (int k = 0; k < nblk; ++k) {
        const uint32_t nb = (uint32_t)(nrow * bw[k] * 8);
        const double* src = bsrc[k] + rb * bld[k];
        if (bld[k] == bw[k] && ((uintptr_t)src & 15) == 0 && (nb & 15) == 0) {
          bytes += nb;
        } else {
          for (int t = lane; t < nrow * bw[k]; t += 32) {
            const int rr = t / bw[k], j = t - rr * bw[k];
            dst0[boff[k] + t] = src[(int64_t)rr * bld[k] + j];
          }
        }
      }
      __syncwarp();
      if (lane == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(BAR(OZ_B_RAWF, rs)), "r"(bytes)
                     : "memory");
        for (int k = 0; k < nblk; ++k) {
          const uint32_t nb = (uint32_t)(nrow * bw[k] * 8);
          const double* src = bsrc[k] + rb * bld[k];
          if (bld[k] == bw[k] && ((uintptr_t)src & 15) == 0 && (nb & 15) == 0 && nb > 0)
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    smem_u32(dst0 + boff[k])),
                "l"(src), "r"(nb), "r"(BAR(OZ_B_RAWF, rs))
                : "memory");
        }
      }
      issued = cc + 1;
    }
    // the copies still in flight land before the CTA may exit
    if (lane == 0)
      for (int cc = max(0, issued - nraw); cc < issued; ++cc)
        if (!mbar_drain(BAR(OZ_B_RAWF, cc % nraw), (uint32_t)(cc / nraw) & 1u)) atomicExch(sflag, 1);
    __syncwarp();
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const bool ok = *(volatile int*)sflag == 0;
  if (!ok && tid == 0) atomicExch(g.status, 1);
  if (warp == OZ_MMA_WARP)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(OZ_TMEM_COLS));
}


// ---- linear combinations O = [A_0 .. A_nb-1] C on the tensor cores --------
//
// O(r, j) = sum_i A(r, i) C(i, j): the Davidson updates (Gram-Schmidt and
// Cholesky-QR, Ritz vectors, re-contraction).  A is nb blocks of nsd columns
// (rows nsd doubles apart, blocks sA apart), C is (m x nsd) row-major
// (m = nb nsd), O has rows ldO doubles apart and may be the last block of A.
// The contraction runs over i, so each row r of A gets its own exponent
// (the largest over its m values) and C one per column j; the digits and
// levels are those of k_gram_oz, and a level of one entry sums at most
// m <= 128 products, below 2^23.
//
// One CTA per SM walks tiles of 128 rows, one role per warp:
//  * the load warp streams the tiles' blocks through a ring of block slots in
//    shared memory (one cp.async.bulk per block, completing on the tile's
//    rawf[t % 2]); a slot is refilled once the K step that read it last is
//    cut, which the MMA warp publishes as it waits for the steps in order, so
//    up to a whole tile is on its way while a tile is cut;
//  * warps 0-15 form the row exponents and cut each K step of 16 columns into
//    the 8 A digit planes of stage s (full[s]); a warp owns 8 rows, its lanes
//    4 columns each, so that a row's exponent is two shuffles and the two
//    16-byte loads of a lane, the second half first in the upper columns,
//    touch every bank once;
//  * the MMA warp issues the step's 8 MMAs (M = 128 rows, N = (8 - p) 16,
//    K = 16) into one of two tensor-memory accumulators and commits them to
//    empty[s] and, at the end of a tile, to accf[b];
//  * four warps read a finished accumulator, add its levels as integers and
//    write the tile's rows of O in FP64 (acce[b]).
// The digit planes of C are built once per CTA.  Waits are bounded as in
// k_gram_oz.  1e6 rows x 80 -> 8 columns: 350 us, against 798 us when all
// warps cut, issued and flushed in turn behind block barriers.  What is left
// (14k cycles a tile): the digit stores and operand reads of shared memory
// (about 1k cycles a K step), the integer instructions of the cut (50 us of
// the time), the exponent pass and the wait for a tile's last blocks (50 us
// each).
constexpr int LC_SPLIT_WARPS = 16;
constexpr int LC_FLUSH_WARP = LC_SPLIT_WARPS;    // a multiple of 4: warp w reads lane quarter w % 4
constexpr int LC_MMA_WARP = LC_FLUSH_WARP + 4;
constexpr int LC_LOAD_WARP = LC_MMA_WARP + 1;
constexpr int LC_THREADS = (LC_LOAD_WARP + 1) * 32;
constexpr int LC_TM = 128;                       // rows per tile (MMA M)
constexpr int LC_KS = 16;                        // K step (columns of A)
constexpr int LC_APLANE = LC_TM * LC_KS * 2;     // 4 KB: one A digit plane of one K step
constexpr int LC_ASTAGE = OZ_DIG * LC_APLANE;    // 32 KB
constexpr int LC_BCHUNK = OZ_DIG * OZ_N * LC_KS * 2;  // 4 KB: the 8 C planes of one K step
constexpr int LC_MAXM = 128;
constexpr int LC_ACC_COLS = OZ_LEVELS * OZ_N;    // 128 tensor-memory columns per accumulator
constexpr int LC_TMEM_COLS = 2 * LC_ACC_COLS;
// barrier slots
constexpr int LC_MAXST = 3;                      // digit stages: 3 where shared memory allows, else 2
constexpr int LC_B_FULL = 0, LC_B_EMPTY = LC_B_FULL + LC_MAXST, LC_B_ACCF = LC_B_EMPTY + LC_MAXST,
              LC_B_ACCE = LC_B_ACCF + 2, LC_B_RAWF = LC_B_ACCE + 2, LC_NBARS = LC_B_RAWF + 2;

struct LcArgs {
  const double* A;
  int64_t sA;
  int m, nsd;
  const double* C;  // (m, nsd) row-major
  double* O;
  int64_t ldO;
  int64_t N, rows_per_cta;
  int lane_copies;  // some block of some tile is not whole 16-byte lines
  int nslots;       // block slots of the ring: nb .. 2 nb
  int nst;          // digit stages
  const int* skip;
  int* status;
};

// byte offset of (row, k) in a K-major tile of 8 x 16-byte core matrices
// with K = 16: row-group stride (SBO) 256 bytes, K-direction stride (LBO) 128
__device__ __forceinline__ int kmaj16(int row, int k) {
  return (((row >> 3) * 2) + (k >> 3)) * 128 + (row & 7) * 16 + (k & 7) * 2;
}
__device__ __forceinline__ uint64_t sdesc16(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) |
         ((uint64_t)1 << 46);
}

__device__ __forceinline__ int biased_exp(double x) { return (int)(((unsigned)__double2hiint(x) >> 20) & 0x7FF); }

// 8 columns of one level (exact integers below 2^23) of this warp's 32 lanes
__device__ __forceinline__ void lc_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}

// VEC: nsd a multiple of 4, so that the four columns of a lane are two 16-byte
// loads of one staged block
template <bool VEC>
__global__ void __launch_bounds__(LC_THREADS, 1) k_lincomb_oz(LcArgs g) {
  if (g.skip && *g.skip) return;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sbase = (uint8_t*)(((uintptr_t)smem + 1023) & ~(uintptr_t)1023);
  uint8_t* adig = sbase;                                  // nst stages of 8 A planes
  const int nst = g.nst;
  uint8_t* bdig = sbase + nst * LC_ASTAGE;                // nks x 8 C planes
  const int m = g.m, nsd = g.nsd, nb = m / nsd;
  const int nks = (m + LC_KS - 1) / LC_KS;
  double* raw = (double*)(bdig + (size_t)nks * LC_BCHUNK);  // [slot][128 rows][nsd]
  const int nslots = g.nslots;
  int* eb = (int*)(raw + (size_t)nslots * nsd * LC_TM);   // [2][128] row exponents of two tiles
  int* ej = eb + 2 * LC_TM;                               // [16] column exponents of C
  uint64_t* bars = (uint64_t*)(((uintptr_t)(ej + OZ_N) + 7) & ~(uintptr_t)7);
  uint32_t* tmem_slot = (uint32_t*)(bars + LC_NBARS);
  int* sflag = (int*)(tmem_slot + 1);
  volatile int* sdone = sflag + 1;                        // K steps cut by all splitting warps
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t bar0 = smem_u32(bars);
  auto BAR = [&](int slot) { return bar0 + 8u * (uint32_t)slot; };

  if (warp == LC_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(LC_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int b = 0; b < LC_NBARS; ++b) {
      const int count = b < LC_B_EMPTY ? LC_SPLIT_WARPS
                        : (b == LC_B_ACCE || b == LC_B_ACCE + 1) ? 4
                        : (b >= LC_B_RAWF && g.lane_copies) ? 33
                                                            : 1;
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(BAR(b)), "r"(count));
    }
    asm volatile("fence.mbarrier_init.release.cluster;");
    *sflag = 0;
    *sdone = 0;
  }
  // C: column exponents, then its digit planes (rows j of plane q at q 16 + j)
  for (int x = tid; x < nks * LC_BCHUNK / 16; x += LC_THREADS) reinterpret_cast<uint4*>(bdig)[x] = make_uint4(0, 0, 0, 0);
  if (warp < OZ_N) {
    int e = 0;
    if (warp < nsd)
      for (int i = lane; i < m; i += 32) e = max(e, biased_exp(g.C[(int64_t)i * nsd + warp]));
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) ej[warp] = e;
  }
  __syncthreads();
  for (int x = tid; x < m * nsd; x += LC_THREADS) {
    const int i = x / nsd, j = x - i * nsd;
    uint32_t d[OZ_DIG];
    oz_digits2(g.C[x], 0.0, ej[j], ej[j], d);
    uint8_t* base = bdig + (size_t)(i / LC_KS) * LC_BCHUNK;
    const int k = i % LC_KS;
#pragma unroll
    for (int q = 0; q < OZ_DIG; ++q) *reinterpret_cast<uint16_t*>(base + kmaj16(q * OZ_N + j, k)) = (uint16_t)d[q];
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the C planes are read by the MMAs
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;

  const int64_t r0 = (int64_t)blockIdx.x * g.rows_per_cta;
  const int64_t r1 = min(r0 + g.rows_per_cta, g.N);
  const int ntile = r1 > r0 ? (int)((r1 - r0 + LC_TM - 1) / LC_TM) : 0;

  if (warp < LC_SPLIT_WARPS) {
    // ---- splitting warps: lane (row rl, columns 4 q .. 4 q + 3 of a step) --
    const int q = lane & 3, r = warp * 8 + (lane >> 2);
    const int swap = q >> 1;
    bool ok = true;
    int s = 0, round = 0;  // digit stage of the next K step, uses of it so far
    int slot0 = 0;         // slot of the tile's first block
    auto block = [&](int b) {
      const int x = slot0 + b;
      return raw + (size_t)(x < nslots ? x : x - nslots) * LC_TM * nsd;
    };
    // walks the columns 4 q, 4 q + 16, ... of row r: load() gives the next four (0 beyond m)
    struct Walk {
      int i, b, s;
    };
    const int b0 = 4 * q / nsd, s0 = 4 * q - b0 * nsd;
    auto load = [&](Walk& at, double (&x)[4]) {
      if constexpr (VEC) {
        if (at.i < m) {
          const double2* p = reinterpret_cast<const double2*>(block(at.b) + r * nsd + at.s);
          const double2 u = p[swap], w = p[1 - swap];
          x[0] = swap ? w.x : u.x;
          x[1] = swap ? w.y : u.y;
          x[2] = swap ? u.x : w.x;
          x[3] = swap ? u.y : w.y;
        } else {
          x[0] = x[1] = x[2] = x[3] = 0.0;
        }
      } else {
        int b = at.b, s = at.s;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          x[k] = 0.0;
          if (at.i + k < m) x[k] = block(b)[r * nsd + s];
          if (++s == nsd) {
            s = 0;
            ++b;
          }
        }
      }
      at.i += LC_KS;
      at.s += LC_KS;
      while (at.s >= nsd) {
        at.s -= nsd;
        ++at.b;
      }
    };
    for (int t = 0; t < ntile && ok; ++t) {
      if (t > 0) slot0 = (slot0 + nb) % nslots;
      ok = mbar_wait(BAR(LC_B_RAWF + (t & 1)), (uint32_t)(t >> 1) & 1u, sflag);
      if (!__all_sync(0xffffffffu, ok)) {
        ok = false;
        break;
      }
      // the row's largest exponent
      int e = 0;
      Walk at{4 * q, b0, s0};
#pragma unroll 2
      for (int c = 0; c < nks; ++c) {
        double x[4];
        load(at, x);
#pragma unroll
        for (int k = 0; k < 4; ++k) e = max(e, __double2hiint(x[k]) & 0x7fffffff);
      }
      at = Walk{4 * q, b0, s0};
      e >>= 20;
      e = max(e, __shfl_xor_sync(0xffffffffu, e, 1));
      e = max(e, __shfl_xor_sync(0xffffffffu, e, 2));
      // tile t - 2 has been written: its exponents may go
      if (t >= 2) ok = mbar_wait(BAR(LC_B_ACCE + (t & 1)), (uint32_t)((t >> 1) - 1) & 1u, sflag);
      if (!__all_sync(0xffffffffu, ok)) {
        ok = false;
        break;
      }
      if (q == 0) eb[(t & 1) * LC_TM + r] = e;
      for (int c = 0; c < nks; ++c) {
        double x[4];
        load(at, x);
        uint32_t d0[OZ_DIG], d1[OZ_DIG];
        oz_digits2(x[0], x[1], e, e, d0);
        oz_digits2(x[2], x[3], e, e, d1);
        // the MMAs of nst steps ago are done with stage s
        if (round > 0) ok = mbar_wait(BAR(LC_B_EMPTY + s), (uint32_t)(round - 1) & 1u, sflag);
        if (!__all_sync(0xffffffffu, ok)) {
          ok = false;
          break;
        }
        uint8_t* dst = adig + s * LC_ASTAGE + kmaj16(r, 4 * q);
#pragma unroll
        for (int p = 0; p < OZ_DIG; ++p) *reinterpret_cast<uint2*>(dst + p * LC_APLANE) = make_uint2(d0[p], d1[p]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR(LC_B_FULL + s));
        if (++s == nst) {
          s = 0;
          ++round;
        }
      }
    }
    if (!ok && lane == 0) atomicExch(sflag, 1);
  } else if (warp < LC_MMA_WARP) {
    // ---- flush warps: lane quarter q = warp % 4 holds rows 32 q .. 32 q + 31
    const int r = (warp & 3) * 32 + lane;
    const uint32_t lrow = (uint32_t)((warp & 3) * 32) << 16;
    const bool o16 = (((uintptr_t)g.O & 15) == 0) && (g.ldO & 1) == 0 && (nsd & 1) == 0;
    for (int t = 0; t < ntile; ++t) {
      const int buf = t & 1;
      const bool ok = mbar_wait(BAR(LC_B_ACCF + buf), (uint32_t)(t >> 1) & 1u, sflag);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) atomicExch(sflag, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t ta = tmem + lrow + (uint32_t)(buf * LC_ACC_COLS);
      const int64_t row = r0 + (int64_t)t * LC_TM + r;
      const int er = eb[buf * LC_TM + r];
      for (int j0 = 0; j0 < nsd; j0 += 8) {
        long long hi[8], lo[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) hi[j] = lo[j] = 0;
#pragma unroll
        for (int L = 0; L < OZ_LEVELS; L += 2) {
          uint32_t v0[8], v1[8];
          lc_ld8(ta + L * OZ_N + j0, v0);
          lc_ld8(ta + (L + 1) * OZ_N + j0, v1);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const long long i0 = (long long)__float2int_rn(__uint_as_float(v0[j]));
            const long long i1 = (long long)__float2int_rn(__uint_as_float(v1[j]));
            if (L < OZ_LEVELS / 2)
              hi[j] += (i0 << (7 * (3 - L))) + (i1 << (7 * (2 - L < 0 ? 0 : 2 - L)));
            else
              lo[j] += (i0 << (7 * (7 - L))) + (i1 << (7 * (6 - L < 0 ? 0 : 6 - L)));
          }
        }
        if (j0 + 8 >= nsd) {  // everything of this accumulator and tile is read
          asm volatile("tcgen05.fence::before_thread_sync;");
          __syncwarp();
          if (lane == 0) mbar_arrive(BAR(LC_B_ACCE + buf));
        }
        if (row < r1) {
          double* o = g.O + row * g.ldO + j0;
          double v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (j0 + j < nsd) {
              const int ex = (er - 1022) + (ej[j0 + j] - 1022);
              if (ex - 63 >= -1022 && ex - 35 <= 960)  // both parts exact, one rounding
                v[j] = scaled_int(hi[j], ex - 35) + scaled_int(lo[j], ex - 63);
              else
                v[j] = ldexp((double)hi[j], ex - 35) + ldexp((double)lo[j], ex - 63);
            }
          }
#pragma unroll
          for (int j = 0; j < 8; j += 2) {
            if (o16) {
              if (j0 + j < nsd) *reinterpret_cast<double2*>(o + j) = make_double2(v[j], v[j + 1]);
            } else {
              if (j0 + j < nsd) o[j] = v[j];
              if (j0 + j + 1 < nsd) o[j + 1] = v[j + 1];
            }
          }
        }
      }
    }
  } else if (warp == LC_MMA_WARP) {
    // ---- MMA warp: lane 0 issues, the warp stays converged ----------------
    uint32_t last_bar = 0, last_par = 0;  // the latest commit: its completion covers every MMA
    int gstep = 0, s = 0, round = 0;
    bool ok = true;
    for (int t = 0; t < ntile && ok; ++t)
      for (int c = 0; c < nks && ok; ++c, ++gstep) {
        const int buf = t & 1;
        if (lane == 0) {
          // accumulator written out (tile t - 2), digit stage s full
          if (c == 0 && t >= 2) ok = mbar_wait(BAR(LC_B_ACCE + buf), (uint32_t)((t >> 1) - 1) & 1u, sflag);
          if (ok) ok = mbar_wait(BAR(LC_B_FULL + s), (uint32_t)round & 1u, sflag);
          if (ok) {
            // every read of this step's slots, which the barrier has put before
            // this thread, comes before their next copies
            __threadfence_block();
            *sdone = gstep + 1;
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t a0 = smem_u32(adig + s * LC_ASTAGE), b0 = smem_u32(bdig + (size_t)c * LC_BCHUNK);
#pragma unroll
            for (int p = 0; p < OZ_DIG; ++p) {
              const uint32_t acc = (c == 0 && p == 0) ? 0u : 1u;
              asm volatile(
                  "{\n .reg .pred pa;\n setp.ne.b32 pa, %4, 0;\n"
                  " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, pa;\n}" ::"r"(
                      tmem + (uint32_t)(buf * LC_ACC_COLS + p * OZ_N)),
                  "l"(sdesc16(a0 + p * LC_APLANE)), "l"(sdesc16(b0)), "r"(oz_idesc((OZ_LEVELS - p) * OZ_N)), "r"(acc));
            }
            mma_commit(BAR(LC_B_EMPTY + s));
            last_bar = BAR(LC_B_EMPTY + s);
            last_par = (uint32_t)round & 1u;
            if (c == nks - 1) mma_commit(BAR(LC_B_ACCF + buf));
          } else {
            atomicExch(sflag, 1);
          }
        }
        if (++s == nst) {
          s = 0;
          ++round;
        }
        ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
      }
    // before the tensor memory is freed, every MMA issued must have completed
    if (lane == 0 && last_bar != 0 && !mbar_drain(last_bar, last_par)) atomicExch(sflag, 1);
    __syncwarp();
  } else {
    // ---- load warp: blocks of tile t in order, each as one bulk copy, or by
    // the lanes when it is not whole 16-byte lines (g.lane_copies: some are not)
    struct Io {
      const LcArgs& g;
      const int* sflag;
      volatile int* sdone;
      int64_t r0, r1;
      int nsd, lane;
      uint32_t rawf;  // barriers of the even and odd tiles
      uint32_t dst0;  // first slot
      const double* tile;  // first block of the tile being loaded, and the bytes of its blocks
      uint32_t bytes;
      __device__ __forceinline__ uint32_t bar(int t) const { return rawf + 8u * (uint32_t)(t & 1); }
      // bounded wait for K step `step` of the whole run to be cut: the steps cut, 0 when it gave up
      __device__ __forceinline__ int cut(int step) const {
        int done = 0;
        for (long long it = 0; it < OZ_WAIT_LIMIT; ++it) {
          done = *sdone;
          if (done > step || ((it & 255) == 255 && *(volatile const int*)sflag)) break;
        }
        __threadfence_block();
        done = __reduce_min_sync(0xffffffffu, done);
        return done > step ? done : 0;
      }
      __device__ __forceinline__ void begin(int t) {
        const int64_t R = r0 + (int64_t)t * LC_TM;
        tile = g.A + R * nsd;
        bytes = (uint32_t)(min((int64_t)LC_TM, r1 - R) * nsd * 8);
      }
      // one bulk copy a block, started by a lane each when there are many, or by
      // all lanes when the block is not whole 16-byte lines
      __device__ __forceinline__ void copy(int t, int b, int n, int slot) const {
        const uint32_t step = (uint32_t)(LC_TM * nsd * 8);
        const double* src = tile + (int64_t)b * g.sA;
        uint32_t dst = dst0 + (uint32_t)slot * step;
        if (n >= 8 && !g.lane_copies) {
          if (lane == 0) expect(t, (uint32_t)n * bytes);
          __syncwarp();
          for (int i = lane; i < n; i += 32) bulk(t, dst + (uint32_t)i * step, src + (int64_t)i * g.sA);
          __syncwarp();
          return;
        }
        for (int i = 0; i < n; ++i, src += g.sA, dst += step) {
          if (!g.lane_copies || (((uintptr_t)src | bytes) & 15) == 0) {
            if (lane == 0) {
              expect(t, bytes);
              bulk(t, dst, src);
            }
          } else {
            for (uint32_t x = lane; x < bytes / 8; x += 32)
              asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 8u * x), "l"(src + x) : "memory");
          }
        }
      }
      __device__ __forceinline__ void expect(int t, uint32_t n) const {
        asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar(t)), "r"(n) : "memory");
      }
      __device__ __forceinline__ void bulk(int t, uint32_t dst, const double* src) const {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                     "l"(src), "r"(bytes), "r"(bar(t))
                     : "memory");
      }
      __device__ __forceinline__ void finish(int t) const {
        if (lane == 0) mbar_arrive(bar(t));
        if (g.lane_copies)  // the lanes' share of the tile arrives once their copies have landed
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar(t)) : "memory");
      }
      __device__ __forceinline__ void drain(int t) const {
        if (lane == 0 && !mbar_drain(bar(t), (uint32_t)(t >> 1) & 1u)) atomicExch(const_cast<int*>(sflag), 1);
      }
    };
    Io io{g, sflag, sdone, r0, r1, nsd, lane, BAR(LC_B_RAWF), smem_u32(raw), nullptr, 0};
    if (!block_ring_load<LC_KS>(io, ntile, nb, nslots, nsd, nks) && lane == 0) atomicExch(sflag, 1);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (tid == 0 && *(volatile int*)sflag) atomicExch(g.status, 1);
  if (warp == LC_MMA_WARP)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(LC_TMEM_COLS));
}

// biased max exponent of each column (nsd <= 256 columns per block, rows ld
// values apart, nblk blocks sX apart) into E[col0 + block * nsd + s]
// (atomicMax; E must be zeroed first).  Thread t of a CTA keeps column
// t % nsd of the CTA's rows t / nsd, + rows per pass, ...: consecutive
// threads read consecutive values of a row.  Order-independent, hence
// deterministic.
__global__ void __launch_bounds__(256) k_col_maxexp(const double* X, int nblk, int64_t sX, int nsd, int ld, int64_t N,
                                                    int* E, int col0, const int* skip) {
  if (skip && *skip) return;
  __shared__ int smax[256];
  const int rpp = blockDim.x / nsd;  // rows per pass of one CTA
  const int c = threadIdx.x % nsd, rl = threadIdx.x / nsd;
  const int64_t rstep = (int64_t)gridDim.x * rpp;
  for (int b = 0; b < nblk; ++b) {
    const double* x = X + (int64_t)b * sX;
    for (int i = threadIdx.x; i < nsd; i += blockDim.x) smax[i] = 0;
    __syncthreads();
    int mx = 0;
    if (rl < rpp) {
#pragma unroll 4
      for (int64_t r = (int64_t)blockIdx.x * rpp + rl; r < N; r += rstep)
        mx = max(mx, (int)(((unsigned long long)__double_as_longlong(x[r * ld + c]) >> 52) & 0x7FF));
      if (mx > 0) atomicMax(&smax[c], mx);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nsd; i += blockDim.x)
      if (smax[i] > 0) atomicMax(&E[col0 + b * nsd + i], smax[i]);
    __syncthreads();
  }
}

// The CTAs' partial sums of one entry per thread, added in the CTAs' order.
// Bound by the latency of the loads, so OZ_RED_AHEAD of them are in flight
// at a time and the entries are spread over one warp per block.
constexpr int OZ_RED_AHEAD = 16;
__global__ void k_oz_reduce(const double* __restrict__ partial, int ncta, int np, double* __restrict__ out,
                            const int* skip) {
  if (skip && *skip) return;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < np; p += gridDim.x * blockDim.x) {
    double s = 0.0;
    int c = 0;
    for (; c + OZ_RED_AHEAD <= ncta; c += OZ_RED_AHEAD) {
      double v[OZ_RED_AHEAD];
#pragma unroll
      for (int i = 0; i < OZ_RED_AHEAD; ++i) v[i] = partial[(int64_t)(c + i) * np + p];
#pragma unroll
      for (int i = 0; i < OZ_RED_AHEAD; ++i) s += v[i];
    }
    for (; c < ncta; ++c) s += partial[(int64_t)c * np + p];
    out[p] = s;
  }
}

}  // namespace

void qp_oz_reduce(const double* partial, int ncta, int np, double* out, const int* skip, cudaStream_t st) {
  k_oz_reduce<<<(np + 31) / 32, 32, 0, st>>>(partial, ncta, np, out, skip);
}

// Opt-in shared memory of k_gram_oz on the current device (once per device).
int qp_gram_oz_prepare() {
  static int done[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  if (done[dev]) return 0;
  if (cudaFuncSetAttribute(k_gram_oz, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM_MAX) != cudaSuccess)
    return -1;
  done[dev] = 1;
  return 0;
}

void qp_col_maxexp(const double* X, int nblk, int64_t sX, int nsd, int ld, int64_t N, int* E, int col0,
                   const int* skip, cudaStream_t st, int n_sm) {
  k_col_maxexp<<<4 * n_sm, 256, 0, st>>>(X, nblk, sX, nsd, ld, N, E, col0, skip);
}

// X (m x nbc, row-major) = A^T [B0 B1] per CTA into partial[cta][m][nbc];
// A: m columns in blocks of nsdA (rows ldA apart, blocks sA apart); B0 (and
// B1): nsdB columns each, rows ldB apart; m <= 128, nbc <= 16.  Exponents eA
// (m), eB (nbc) from qp_col_maxexp.
void qp_gram_oz(const double* A, int64_t sA, int m, int nsdA, int ldA, const double* B0, const double* B1, int nbc,
                int nsdB, int ldB, int64_t N, const int* eA, const int* eB, double* partial, int ncta,
                const int* skip, int* status, cudaStream_t st) {
  OzArgs g;
  g.A = A;
  g.sA = sA;
  g.m = m;
  g.nsdA = nsdA;
  g.ldA = ldA;
  g.B0 = B0;
  g.B1 = B1;
  g.nbc = nbc;
  g.nsdB = nsdB;
  g.ldB = ldB;
  g.N = N;
  int64_t rpc = (N + ncta - 1) / ncta;
  rpc = (rpc + OZ_KC - 1) / OZ_KC * OZ_KC;
  g.rows_per_cta = rpc;
  g.eA = eA;
  g.eB = eB;
  g.partial = partial;
  g.skip = skip;
  g.status = status;
  // raw stages of OZ_KC rows of the m + nbc columns (256-byte aligned): as
  // many as fit beside the digit stages, up to OZ_MAXRAW
  const int rw = m + nbc;
  g.raw_stride = (OZ_KC * rw + 31) / 32 * 32;
  // digit stages of the columns in use; the MMAs of the last stage read up to
  // 128 rows of its last A plane, inside its B planes and the raw stages
  g.a_tile = (m + 7) / 8 * 8 * OZ_KC * 2;
  g.stage = OZ_DIG * (g.a_tile + OZ_B_TILE);
  auto rawfit = [&](int nst) { return (OZ_SMEM_MAX - nst * g.stage - OZ_TAB) / (g.raw_stride * 8); };
  g.nst = rawfit(3) >= 2 ? 3 : 2;
  g.nraw = std::max(1, std::min(OZ_MAXRAW, rawfit(g.nst)));
  const int smem = g.nst * g.stage + g.nraw * g.raw_stride * 8 + OZ_TAB;
  // rows per splitting task, by what each measured over 2 to 144 columns: wide
  // tasks need the fewest stores, narrow ones the shortest chain when a chunk
  // leaves most splitting threads without one.  1e6 rows, 2 / 4 / 8 rows: 4 + 4
  // columns 250 / 256 / 260 us, 8 + 4 281 / 270 / 270, 8 + 8 292 / 280 / 281,
  // 16 + 1 309 / 305 / 281, 48 + 4 448 / 412 / 378, 128 + 16 874 / 768 / 702
  g.rpt = rw <= 8 ? 2 : rw <= 16 ? 4 : 8;
  g.nsw = std::min(OZ_SPLIT / 32, (rw * (OZ_KC / g.rpt) + 31) / 32);
  k_gram_oz<<<ncta, OZ_THREADS, smem, st>>>(g);
}


// Opt-in shared memory of k_lincomb_oz (once per device).
static int lincomb_oz_prepare() {
  static int done[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  if (done[dev]) return 0;
  if (cudaFuncSetAttribute(k_lincomb_oz<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM_MAX) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_lincomb_oz<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM_MAX) !=
          cudaSuccess)
    return -1;
  done[dev] = 1;
  return 0;
}

// O = [A_0 .. A_nb-1] C on the tensor cores (FP64-accurate); m = nb nsd <=
// 128, nsd <= 16.  Returns -1 when the shapes are outside the kernel's range
// (the caller keeps its FP64 path), else 0.
int qp_lincomb_oz(const double* A, int64_t sA, int m, int nsd, const double* C, double* O, int64_t ldO, int64_t N,
                  int ncta, const int* skip, int* status, cudaStream_t st) {
  if (m < 1 || m > LC_MAXM || nsd < 1 || nsd > OZ_N || m % nsd) return -1;
  if (lincomb_oz_prepare()) return -1;
  const int nks = (m + LC_KS - 1) / LC_KS;
  const int nb = m / nsd;
  // three digit stages where a quarter of a tile can still be loaded ahead
  const size_t slot_bytes = (size_t)LC_TM * nsd * 8;
  auto fixed = [&](int nst) {
    return 1024 + (size_t)nst * LC_ASTAGE + (size_t)nks * LC_BCHUNK + (2 * LC_TM + OZ_N) * 4 + (LC_NBARS + 3) * 8;
  };
  const int nst = fixed(3) + (nb + (nb + 3) / 4) * slot_bytes <= (size_t)OZ_SMEM_MAX ? 3 : 2;
  const int nslots = std::min<int>(2 * nb, (int)((OZ_SMEM_MAX - fixed(nst)) / slot_bytes));
  if (nslots < nb) return -1;
  const size_t smem = fixed(nst) + nslots * slot_bytes;
  LcArgs g;
  g.A = A;
  g.sA = sA;
  g.m = m;
  g.nsd = nsd;
  g.C = C;
  g.O = O;
  g.ldO = ldO;
  g.N = N;
  int64_t rpc = (N + ncta - 1) / ncta;
  rpc = (rpc + LC_TM - 1) / LC_TM * LC_TM;
  g.rows_per_cta = rpc;
  g.nslots = nslots;
  g.nst = nst;
  // blocks start on 16-byte lines, and the last tile's rows fill them
  g.lane_copies = ((uintptr_t)A & 15) != 0 || (nb > 1 && (sA & 1) != 0) || ((N % LC_TM) * nsd & 1) != 0;
  g.skip = skip;
  g.status = status;
  if ((nsd & 3) == 0)
    k_lincomb_oz<true><<<ncta, LC_THREADS, smem, st>>>(g);
  else
    k_lincomb_oz<false><<<ncta, LC_THREADS, smem, st>>>(g);
  return 0;
}

extern "C" int qpgpu_gram_tc(qpgpu_ctx* c, const double* A, int64_t lda, int m, const double* B, int64_t ldb, int n,
                             int64_t N, double* X, void* stream) {
  if (!c) return QPGPU_ERR_ARG;
  if (!A || !B || !X || m < 1 || m > 128 || n < 1 || n > 16 || N < 1 || lda < m || ldb < n || lda > (1 << 30) ||
      ldb > (1 << 30))
    return qpgpu_fail(c, QPGPU_ERR_ARG, "gram_tc: need 1 <= m <= 128, 1 <= n <= 16, N >= 1, lda >= m, ldb >= n");
  std::lock_guard<std::mutex> lk(c->mu);
  if (qp_gram_oz_prepare()) return qpgpu_fail(c, QPGPU_ERR_CUDA, "gram_tc: shared-memory opt-in failed");
  const int ncta = c->n_sm;
  const size_t need = (size_t)ncta * m * n * sizeof(double) + (size_t)(m + n + 8) * sizeof(int) + 256;
  if (c->tc_scratch_bytes < need) {
    dev_free(c, c->d_tc_scratch);
    c->d_tc_scratch = nullptr;
    c->tc_scratch_bytes = 0;
    QP_CUDA(c, qp_dev_malloc(c, &c->d_tc_scratch, need));
    c->tc_scratch_bytes = need;
  }
  double* part = (double*)c->d_tc_scratch;
  int* E = (int*)(part + (size_t)ncta * m * n);
  int* status = E + m + n;
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  QP_CUDA(c, cudaMemsetAsync(E, 0, (m + n + 1) * sizeof(int), st));
  qp_col_maxexp(A, 1, 0, m, (int)lda, N, E, 0, nullptr, st, c->n_sm);
  qp_col_maxexp(B, 1, 0, n, (int)ldb, N, E + m, 0, nullptr, st, c->n_sm);
  qp_gram_oz(A, 0, m, m, (int)lda, B, nullptr, n, n, (int)ldb, N, E, E + m, part, ncta, nullptr, status, st);
  qp_oz_reduce(part, ncta, m * n, X, nullptr, st);
  int hs = 0;
  QP_CUDA(c, cudaMemcpyAsync(&hs, status, sizeof(int), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaStreamSynchronize(st));
  if (hs) return qpgpu_fail(c, QPGPU_ERR_TIMEOUT, "gram_tc: a bounded tensor-core wait ran out");
  return QPGPU_OK;
}

extern "C" int qpgpu_lincomb_tc(qpgpu_ctx* c, const double* A, int64_t sA, int m, int nsd, const double* C, double* O,
                                int64_t ldO, int64_t N, void* stream) {
  if (!c) return QPGPU_ERR_ARG;
  if (!A || !C || !O || m < 1 || m > LC_MAXM || nsd < 1 || nsd > OZ_N || m % nsd || N < 1 || ldO < nsd ||
      (m > nsd && sA < N * nsd))
    return qpgpu_fail(c, QPGPU_ERR_ARG, "lincomb_tc: need m = nb nsd <= 128, nsd <= 16, N >= 1, ldO >= nsd, sA >= N nsd");
  std::lock_guard<std::mutex> lk(c->mu);
  if (!c->d_tc_scratch || c->tc_scratch_bytes < sizeof(int)) {
    dev_free(c, c->d_tc_scratch);
    c->d_tc_scratch = nullptr;
    c->tc_scratch_bytes = 0;
    QP_CUDA(c, qp_dev_malloc(c, &c->d_tc_scratch, 256));
    c->tc_scratch_bytes = 256;
  }
  int* status = (int*)c->d_tc_scratch;
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  QP_CUDA(c, cudaMemsetAsync(status, 0, sizeof(int), st));
  if (qp_lincomb_oz(A, sA, m, nsd, C, O, ldO, N, c->n_sm, nullptr, status, st))
    return qpgpu_fail(c, QPGPU_ERR_CUDA, "lincomb_tc: shared-memory opt-in failed");
  QP_CUDA(c, cudaGetLastError());
  int hs = 0;
  QP_CUDA(c, cudaMemcpyAsync(&hs, status, sizeof(int), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaStreamSynchronize(st));
  if (hs) return qpgpu_fail(c, QPGPU_ERR_TIMEOUT, "lincomb_tc: a bounded tensor-core wait ran out");
  return QPGPU_OK;
}
