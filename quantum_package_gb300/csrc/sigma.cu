// Sigma application v = H u, s = S^2 u over the stored connected pairs.
//
// The reference computes every matrix element again at each call
// (src/Davidson/u0Hu0.irp.f:177-444); here they are built once per
// determinant set and sigma is a row-owner gather: each row is owned by one
// warp (rows longer than CHUNK pairs are split over several warps whose
// partial sums are added in a fixed order), so there are no atomics and the
// result is deterministic.  u is laid out (N_det, N_st) with states fastest,
// as u_t(N_st, N_det) in the reference (:27-41), so the N_st coefficients of a
// connected determinant J are one contiguous load.
#include <algorithm>
#include <cstdio>

#include <cub/cub.cuh>

#include "qpgpu_internal.cuh"
#include "sigma_device.cuh"

namespace {

constexpr int SBLK = 256;

struct SigArgs {
  int64_t N;
  const int64_t* rowptr;
  const int* colidx;
  const double* val64;
  const float* val32;
  const int64_t* s2ptr;
  const int* s2col;
  const float* s2val;
  const double* hdiag;
  const double* sdiag;
  const int* item_row;
  const int* item_sub;
  const int* row_nitems;
  int64_t n_items;
  const double* u;   // (N, NST) FP64
  const float* u32;  // (N, u32_ld) FP32 (precision FP32): rows u32_ld floats apart
  int u32_ld;
  const float* u32lo;   // precision FF: low parts of u, same layout as u32 (the high parts)
  const float* val32lo; // precision FF: low parts of the stored elements (val32 = high parts)
  double* v;
  double* s;
  double* pv;  // partial sums (n_items, NST)
  double* ps;
  int row_lo, row_hi;  // rows [row_lo, row_hi) are written (range variant)
  int row_step, row_first;
};

__device__ __forceinline__ bool row_selected(const SigArgs& a, int k) {
  if (k < a.row_lo || k >= a.row_hi) return false;
  return ((k - a.row_first) % a.row_step) == 0;
}

using namespace qpsig;

// write the reduced state sums (lane L holds state L >> shift) and the
// diagonal: of each state's lanes the first does v, the second s, in one FP64
// instruction
template <int NST>
__device__ __forceinline__ void store_row(const SigArgs& a, int64_t it, int k, int lane, double hv, double sv,
                                          bool has_s2) {
  constexpr int SH = 5 - Pow2<NST>::lg;
  const int st = lane >> SH, sub = lane & ((1 << SH) - 1);
  if (sub > 1 || st >= NST) return;
  const double sum = sub == 0 ? hv : has_s2 ? sv : 0.0;
  if (a.row_nitems[k] == 1) {
    const double d = __ldg(sub == 0 ? &a.hdiag[k] : &a.sdiag[k]);
    (sub == 0 ? a.v : a.s)[(int64_t)k * NST + st] = fma(d, a.u[(int64_t)k * NST + st], sum);
  } else {
    (sub == 0 ? a.pv : a.ps)[it * NST + st] = sum;
  }
}
// the same by one lane of each state, for the kernels that the FP64 pipe does
// not bound: k_sigma32 keeps 40 instead of 48 registers (1e6 determinants x 4
// states 2.69 -> 2.60 ms)
template <int NST>
__device__ __forceinline__ void store_row_lean(const SigArgs& a, int64_t it, int k, int lane, double hv, double sv,
                                               bool has_s2) {
  constexpr int SH = 5 - Pow2<NST>::lg;
  const int st = lane >> SH;
  if ((lane & ((1 << SH) - 1)) != 0 || st >= NST) return;
  const double s2 = has_s2 ? sv : 0.0;
  if (a.row_nitems[k] == 1) {
    const double uk = a.u[(int64_t)k * NST + st];
    a.v[(int64_t)k * NST + st] = fma(a.hdiag[k], uk, hv);
    a.s[(int64_t)k * NST + st] = fma(a.sdiag[k], uk, s2);
  } else {
    a.pv[it * NST + st] = hv;
    a.ps[it * NST + st] = s2;
  }
}



constexpr int UNR = 4;    // FP64 sigma: pairs per lane per loop trip
constexpr int UNR32 = 4;  // FP32 sigma

// FP64 sigma.  From 3 states on it is bound by the FP64 pipe: an instruction of
// a warp takes 64 cycles of its scheduler's pipe, against one for the integer
// work beside it, so what is not a product is kept off the pipe (empty groups
// of the last trip, conversions of the +-1 of S^2, zeros added in its
// reduction, a second instruction for the diagonal).  With fewer states the
// gathers' latency bounds it, hence four pairs in flight per lane and
// registers for 5 or 6 blocks of an SM.  1e6 determinants x 4 states: 7.42 ->
// 7.27 ms; 2e5 x 1, 2, 3, 4, 8: 287, 390, 512, 626, 1161 -> 244, 359, 489,
// 608, 1142 us.  (256-bit gathers, rows of 3 and 5-7 states padded for them,
// changed that by -1 to +3 percent; six pairs in flight or 8 blocks gain
// nothing but at 2 states.)
template <int NST>
__global__ void __launch_bounds__(SBLK, NST == 1 ? 6 : 5) k_sigma64(SigArgs a) {
  constexpr int NP = Pow2<NST>::v;
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * SBLK + threadIdx.x) >> 5;
  const int64_t nwarp = ((int64_t)gridDim.x * SBLK) >> 5;
  for (int64_t it = warp; it < a.n_items; it += nwarp) {
    const int k = a.item_row[it];
    if (!row_selected(a, k)) continue;
    const int j = a.item_sub[it];
    const int64_t rb = a.rowptr[k], re = a.rowptr[k + 1];
    const int64_t beg = rb + (int64_t)j * QP_SIGMA_CHUNK;
    const int64_t end = min(beg + (int64_t)QP_SIGMA_CHUNK, re);
    double acc[NP];
#pragma unroll
    for (int st = 0; st < NP; ++st) acc[st] = 0.0;
    sum_pairs64<NST, NP, UNR>(a.u, a.colidx, a.val64, beg, end, k, lane, acc);
    const double hsum = reduce_scatter64<NP>(acc, lane);
    double ssum = 0.0;
    const int64_t sb = a.s2ptr[k], se = a.s2ptr[k + 1];
    const bool has_s2 = (j == 0) && (se > sb);
    if (has_s2) {
      ssum = s2_row_sum<NST, NP>(a.u, a.s2col, a.s2val, sb, se, lane);
    }
    store_row<NST>(a, it, k, lane, hsum, ssum, has_s2);
  }
}

// (column, value) pairs of one trip: lane's pairs e0, e0+32, ...; past the
// end of the chunk the row's own column with value 0 (a harmless gather)
__device__ __forceinline__ void load_trip32(const SigArgs& a, int64_t e0, int64_t end, int k, int (&col)[UNR32],
                                            float (&hv)[UNR32]) {
#pragma unroll
  for (int q = 0; q < UNR32; ++q) {
    const int64_t e = e0 + 32 * q;
    col[q] = e < end ? __ldg(&a.colidx[e]) : k;
    hv[q] = e < end ? __ldg(&a.val32[e]) : 0.f;
  }
}

// Kahan-compensated sum += hv * u32[col] for the trip's pairs
template <int NST, int NP, int LD, bool V8>
__device__ __forceinline__ void accumulate32(const SigArgs& a, const int (&col)[UNR32], const float (&hv)[UNR32],
                                             float (&sum)[NP], float (&cmp)[NP]) {
#pragma unroll
  for (int q = 0; q < UNR32; ++q) {
    float x[NST];
    load_row_ld<NST, LD, V8>(a.u32, col[q], x);
#pragma unroll
    for (int st = 0; st < NST; ++st) {
      const float y = __fmaf_rn(hv[q], x[st], -cmp[st]);
      const float t = __fadd_rn(sum[st], y);
      cmp[st] = __fsub_rn(__fsub_rn(t, sum[st]), y);
      sum[st] = t;
    }
  }
}

// FP32 matrix elements x FP32 coefficients with Kahan-compensated lane sums;
// lanes are combined as float-float pairs, and only the owner lane of each
// state converts to FP64 and adds the FP64 diagonal term.
//
// The kernel is bound by the L1TEX data pipe, at 76-81 percent of its peak with
// 4 and 8 states: a wavefront for each distinct 32-byte sector of a coefficient
// gather (2e5 x 8: 309 us; 1e6 x 8: 3.45 ms, with 8 instead of 4 gathers in
// flight 3.52).  With PIPE the next trip's (column, value) pairs are loaded one
// trip ahead of the current trip's gathers, at the price of registers, hence
// occupancy; which launch shape keeps that pipe fed best depends on the row
// lengths, so it is chosen by timing (tune_sigma32).  Every shape gives
// bit-identical sums: each lane sees the same pairs in the same order.
template <int NST, bool PIPE, int BS, int LD, bool V8>
__global__ void __launch_bounds__(BS) k_sigma32(SigArgs a) {
  constexpr int NP = Pow2<NST>::v;
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * BS + threadIdx.x) >> 5;
  const int64_t nwarp = ((int64_t)gridDim.x * BS) >> 5;
  for (int64_t it = warp; it < a.n_items; it += nwarp) {
    const int k = a.item_row[it];
    if (!row_selected(a, k)) continue;
    const int j = a.item_sub[it];
    const int64_t rb = a.rowptr[k], re = a.rowptr[k + 1];
    const int64_t beg = rb + (int64_t)j * QP_SIGMA_CHUNK;
    const int64_t end = min(beg + (int64_t)QP_SIGMA_CHUNK, re);
    float sum[NP], cmp[NP];
#pragma unroll
    for (int st = 0; st < NP; ++st) sum[st] = cmp[st] = 0.f;
    int col[UNR32];
    float hv[UNR32];
    if (PIPE) load_trip32(a, beg + lane, end, k, col, hv);
    for (int64_t e0 = beg + lane; e0 < end; e0 += 32 * UNR32) {
      if (PIPE) {
        int ncol[UNR32];
        float nhv[UNR32];
        load_trip32(a, e0 + 32 * UNR32, end, k, ncol, nhv);
        accumulate32<NST, NP, LD, V8>(a, col, hv, sum, cmp);
#pragma unroll
        for (int q = 0; q < UNR32; ++q) {
          col[q] = ncol[q];
          hv[q] = nhv[q];
        }
        continue;
      }
      load_trip32(a, e0, end, k, col, hv);
#pragma unroll
      for (int q = 0; q < UNR32; ++q) {
        float x[NST];
        load_row_ld<NST, LD, V8>(a.u32, col[q], x);
#pragma unroll
        for (int st = 0; st < NST; ++st) {
          const float y = __fmaf_rn(hv[q], x[st], -cmp[st]);
          const float t = __fadd_rn(sum[st], y);
          cmp[st] = __fsub_rn(__fsub_rn(t, sum[st]), y);
          sum[st] = t;
        }
      }
    }
    // Kahan state (sum, -cmp) is a float-float value
#pragma unroll
    for (int st = 0; st < NP; ++st) cmp[st] = -cmp[st];
    float rh, rl;
    reduce_scatter_ff<NP>(sum, cmp, lane, rh, rl);
    const double hsum = (double)rh + (double)rl;
    double ssum = 0.0;
    const int64_t sb = a.s2ptr[k], se = a.s2ptr[k + 1];
    const bool has_s2 = (j == 0) && (se > sb);
    if (has_s2) {
      float sh[NP], sl[NP];
#pragma unroll
      for (int st = 0; st < NP; ++st) sh[st] = sl[st] = 0.f;
      for (int64_t e = sb + lane; e < se; e += 32) {
        const float sv = __ldg(&a.s2val[e]);  // +-1: products are exact
        float x[NST];
        load_row_ld<NST, LD, V8>(a.u32, __ldg(&a.s2col[e]), x);
#pragma unroll
        for (int st = 0; st < NST; ++st) {
          float s, err;
          two_sum(sh[st], sv * x[st], s, err);
          sh[st] = s;
          sl[st] = __fadd_rn(sl[st], err);
        }
      }
      float qh, ql;
      reduce_scatter_ff<NP>(sh, sl, lane, qh, ql);
      ssum = (double)qh + (double)ql;
    }
    store_row_lean<NST>(a, it, k, lane, hsum, ssum, has_s2);
  }
}

// rows split over several items: add the partials in item order
__global__ void k_sigma_combine(SigArgs a, const int* multi_rows, const int* row_item0, int n_multi, int nst) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < (int64_t)n_multi * nst;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int k = multi_rows[t / nst];
    const int st = (int)(t % nst);
    if (!row_selected(a, k)) continue;
    const int i0 = row_item0[k], ni = a.row_nitems[k];
    double av = 0.0, as = 0.0;
    for (int i = 0; i < ni; ++i) {
      av += a.pv[(int64_t)(i0 + i) * nst + st];
      as += a.ps[(int64_t)(i0 + i) * nst + st];
    }
    const double uk = a.u[(int64_t)k * nst + st];
    a.v[(int64_t)k * nst + st] = fma(a.hdiag[k], uk, av);
    a.s[(int64_t)k * nst + st] = fma(a.sdiag[k], uk, as);
  }
}

// ---- work items -----------------------------------------------------------
// nit[N] = split[N] = 0 (the prefix sums end with the totals)
__global__ void k_row_nitems(const int64_t* rowptr, int* nit, int* split, int64_t N) {
  if (blockIdx.x == 0 && threadIdx.x == 0) nit[N] = split[N] = 0;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < N; k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t nnz = rowptr[k + 1] - rowptr[k];
    const int n = (int)max((int64_t)1, (nnz + QP_SIGMA_CHUNK - 1) / QP_SIGMA_CHUNK);
    nit[k] = n;
    split[k] = n > 1;
  }
}

__global__ void k_fill_items(const int* nit, const int* item0, const int* split0, int* item_row, int* item_sub,
                             int* multi_rows, int64_t N) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < N; k += (int64_t)gridDim.x * blockDim.x) {
    for (int j = 0; j < nit[k]; ++j) {
      item_row[item0[k] + j] = (int)k;
      item_sub[item0[k] + j] = j;
    }
    if (nit[k] > 1) multi_rows[split0[k]] = (int)k;
  }
}

// A thread per determinant d: the columns are read and written in order, and
// the row of d at its position is one or two 32-byte sectors of the L2 (with a
// thread per value in bilinear order each column access moved a sector for 8
// bytes: 30 and 2 x 42 us at 1e6 x 4, now 15 and 28 us).
// bad (optional): set to 1 when an input coefficient is NaN or infinite.
template <int NST>
__global__ void k_to_bilinear(const double* u0, int64_t ld, const int* pos, double* ut, float* ut32, int64_t N,
                              int* bad) {
  for (int64_t d = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; d < N; d += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = pos[d];
    double x[NST];
#pragma unroll
    for (int st = 0; st < NST; ++st) x[st] = u0[(int64_t)st * ld + d];
    if (bad) {
      bool fin = true;
#pragma unroll
      for (int st = 0; st < NST; ++st) fin = fin && isfinite(x[st]);
      if (!fin) *bad = 1;
    }
    double* const r = ut + p * NST;
    if constexpr (NST % 2 == 0) {
#pragma unroll
      for (int st = 0; st < NST; st += 2) *reinterpret_cast<double2*>(r + st) = make_double2(x[st], x[st + 1]);
    } else {
#pragma unroll
      for (int st = 0; st < NST; ++st) r[st] = x[st];
    }
    if (!ut32) continue;
    float* const r32 = ut32 + p * NST;
    if constexpr (NST % 4 == 0) {
#pragma unroll
      for (int st = 0; st < NST; st += 4)
        *reinterpret_cast<float4*>(r32 + st) =
            make_float4((float)x[st], (float)x[st + 1], (float)x[st + 2], (float)x[st + 3]);
    } else {
#pragma unroll
      for (int st = 0; st < NST; ++st) r32[st] = (float)x[st];
    }
  }
}

template <int NST>
__global__ void k_from_bilinear(const double* vt, const double* wt, int64_t ld, const int* pos, double* v0,
                                double* w0, int64_t N) {
  for (int64_t d = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; d < N; d += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = pos[d];
    double x[NST], y[NST];
#pragma unroll
    for (int st = 0; st < NST; ++st) x[st] = vt[p * NST + st];
    if (wt) {
#pragma unroll
      for (int st = 0; st < NST; ++st) y[st] = wt[p * NST + st];
    }
#pragma unroll
    for (int st = 0; st < NST; ++st) v0[(int64_t)st * ld + d] = x[st];
    if (wt) {
#pragma unroll
      for (int st = 0; st < NST; ++st) w0[(int64_t)st * ld + d] = y[st];
    }
  }
}

__global__ void k_nonfinite(const double* x, int64_t n, int* bad) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (!isfinite(x[i])) *bad = 1;
}

// y (N rows of ld floats) <- x (N rows of nst doubles)
// lo = val64 - val32 rounded to FP32 (the low parts of the stored elements)
__global__ void k_lo_parts(const double* v64, const float* v32, float* lo, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    lo[i] = (float)(v64[i] - (double)v32[i]);
}

// (hi, lo) rows of ld floats <- x (N rows of nst doubles), integer split
__global__ void k_split_rows(const double* x, float* hi, float* lo, int64_t N, int nst, int ld) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N * nst; i += (int64_t)gridDim.x * blockDim.x) {
    float h, l;
    split_ff(x[i], h, l);
    const int64_t o = (i / nst) * ld + i % nst;
    hi[o] = h;
    lo[o] = l;
  }
}

__global__ void k_to_float(const double* x, float* y, int64_t N, int nst, int ld) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N * nst; i += (int64_t)gridDim.x * blockDim.x)
    y[(i / nst) * ld + i % nst] = (float)x[i];
}

inline unsigned gsz(int64_t n, int tpb) {
  int64_t g = (n + tpb - 1) / tpb;
  if (g < 1) g = 1;
  if (g > 65535LL * 32) g = 65535LL * 32;
  return (unsigned)g;
}

// FP32 launch shapes tried by the tuner, one warp per work item: CTA size, the
// last one with the next trip's loads ahead
constexpr int kSig32Block[] = {256, 128, 64, 256};
constexpr int kNSig32Shapes = sizeof(kSig32Block) / sizeof(kSig32Block[0]);

template <int NST, int LD, bool V8>
void launch_sigma32_ld(const SigArgs& a, int variant, cudaStream_t st) {
  const unsigned grid = gsz(a.n_items * 32, kSig32Block[variant]);
  switch (variant) {
    case 1: k_sigma32<NST, false, 128, LD, V8><<<grid, 128, 0, st>>>(a); break;
    case 2: k_sigma32<NST, false, 64, LD, V8><<<grid, 64, 0, st>>>(a); break;
    case 3: k_sigma32<NST, true, 256, LD, V8><<<grid, 256, 0, st>>>(a); break;
    default: k_sigma32<NST, false, 256, LD, V8><<<grid, 256, 0, st>>>(a); break;
  }
}

// dense rows (u32_ld == NST) or rows padded to 4 / 8 floats; rows of 8 floats
// on a 32-byte aligned array are read with one 256-bit load each
template <int NST>
void launch_sigma32(const SigArgs& a, int variant, cudaStream_t st) {
  constexpr int P = Pow2<NST>::v;
  const bool a32 = ((uintptr_t)a.u32 & 31) == 0;
  if constexpr (P == 8) {
    if (a.u32_ld == 8 && a32) {
      launch_sigma32_ld<NST, 8, true>(a, variant, st);
      return;
    }
    if constexpr (NST == 8) {
      k_sigma32<8, false, 256, 8, false><<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(
                                               (a.n_items * 32 + 255) / 256, 65535LL * 32)),
                                           256, 0, st>>>(a);
      return;
    }
  }
  if constexpr (P != NST && P == 4) {
    if (a.u32_ld == 4) {
      launch_sigma32_ld<NST, 4, false>(a, variant, st);
      return;
    }
  }
  if constexpr (NST != 8) launch_sigma32_ld<NST, NST, false>(a, variant, st);
}

// Float-float sigma: elements h = vh + vl and coefficients u = uh + ul as
// FP32 pairs (rows padded to LD floats, 32-byte aligned; LD = 8 uses one
// 256-bit load per part).  Per pair and state the product is formed exactly
// for vh*uh (FMA gives its rounding error) plus the cross terms, and each
// lane keeps its sum as an unevaluated float pair updated with Knuth's
// TwoSum; lanes are combined with reduce_scatter_ff.  About 1e-13 relative,
// FP32 pipes only, except the FP64 diagonal term of the owner lanes.
template <int NST, int LD>
__global__ void __launch_bounds__(128) k_sigma_ff(SigArgs a) {
  constexpr int NP = Pow2<NST>::v;
  constexpr int UNRF = 2;
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * 128 + threadIdx.x) >> 5;
  const int64_t nwarp = ((int64_t)gridDim.x * 128) >> 5;
  for (int64_t it = warp; it < a.n_items; it += nwarp) {
    const int k = a.item_row[it];
    if (!row_selected(a, k)) continue;
    const int j = a.item_sub[it];
    const int64_t rb = a.rowptr[k], re = a.rowptr[k + 1];
    const int64_t beg = rb + (int64_t)j * QP_SIGMA_CHUNK;
    const int64_t end = min(beg + (int64_t)QP_SIGMA_CHUNK, re);
    float ah[NP], al[NP];
#pragma unroll
    for (int st = 0; st < NP; ++st) ah[st] = al[st] = 0.f;
    for (int64_t e0 = beg + lane; e0 < end; e0 += 32 * UNRF) {
      int col[UNRF];
      float vh[UNRF], vl[UNRF];
#pragma unroll
      for (int q = 0; q < UNRF; ++q) {
        const int64_t e = e0 + 32 * q;
        col[q] = e < end ? __ldg(&a.colidx[e]) : k;
        vh[q] = e < end ? __ldg(&a.val32[e]) : 0.f;
        vl[q] = e < end ? __ldg(&a.val32lo[e]) : 0.f;
      }
#pragma unroll
      for (int q = 0; q < UNRF; ++q) {
        float xh[NST], xl[NST];
        load_row_ld<NST, LD, LD == 8>(a.u32, col[q], xh);
        load_row_ld<NST, LD, LD == 8>(a.u32lo, col[q], xl);
#pragma unroll
        for (int st = 0; st < NST; ++st) {
          const float p = __fmul_rn(vh[q], xh[st]);
          float pe = __fmaf_rn(vh[q], xh[st], -p);
          pe = __fmaf_rn(vh[q], xl[st], pe);
          pe = __fmaf_rn(vl[q], xh[st], pe);
          float t, err;
          two_sum(ah[st], p, t, err);
          ah[st] = t;
          al[st] = __fadd_rn(al[st], __fadd_rn(err, pe));
        }
      }
    }
    float rh, rl;
    reduce_scatter_ff<NP>(ah, al, lane, rh, rl);
    const double hsum = (double)rh + (double)rl;
    double ssum = 0.0;
    const int64_t sb = a.s2ptr[k], se = a.s2ptr[k + 1];
    const bool has_s2 = (j == 0) && (se > sb);
    if (has_s2) {
      float sh[NP], sl[NP];
#pragma unroll
      for (int st = 0; st < NP; ++st) sh[st] = sl[st] = 0.f;
      for (int64_t e = sb + lane; e < se; e += 32) {
        const float sv = __ldg(&a.s2val[e]);  // +-1: the products are exact
        const int cj = __ldg(&a.s2col[e]);
        float xh[NST], xl[NST];
        load_row_ld<NST, LD, LD == 8>(a.u32, cj, xh);
        load_row_ld<NST, LD, LD == 8>(a.u32lo, cj, xl);
#pragma unroll
        for (int st = 0; st < NST; ++st) {
          float t, err;
          two_sum(sh[st], sv * xh[st], t, err);
          sh[st] = t;
          sl[st] = __fadd_rn(sl[st], __fadd_rn(err, sv * xl[st]));
        }
      }
      float qh, ql;
      reduce_scatter_ff<NP>(sh, sl, lane, qh, ql);
      ssum = (double)qh + (double)ql;
    }
    store_row_lean<NST>(a, it, k, lane, hsum, ssum, has_s2);
  }
}

template <int NST>
void launch_sigma(const SigArgs& a, int precision, unsigned grid, cudaStream_t st, int variant) {
  constexpr int P = Pow2<NST>::v;
  if (precision == QPGPU_FF) {
    const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((a.n_items * 32 + 127) / 128, 65535LL * 32));
    k_sigma_ff<NST, P><<<g, 128, 0, st>>>(a);
  } else if (precision == QPGPU_FP32)
    launch_sigma32<NST>(a, variant < 0 ? 0 : variant, st);
  else
    k_sigma64<NST><<<grid, SBLK, 0, st>>>(a);
}

void launch_any(const SigArgs& a, int nst, int precision, unsigned grid, cudaStream_t st, int variant) {
  switch (nst) {
    case 1: launch_sigma<1>(a, precision, grid, st, variant); break;
    case 2: launch_sigma<2>(a, precision, grid, st, variant); break;
    case 3: launch_sigma<3>(a, precision, grid, st, variant); break;
    case 4: launch_sigma<4>(a, precision, grid, st, variant); break;
    case 5: launch_sigma<5>(a, precision, grid, st, variant); break;
    case 6: launch_sigma<6>(a, precision, grid, st, variant); break;
    case 7: launch_sigma<7>(a, precision, grid, st, variant); break;
    default: launch_sigma<8>(a, precision, grid, st, variant); break;
  }
}

// Times every FP32 launch shape on this determinant set (two launches each,
// the second timed with events on the caller's stream) and keeps the fastest
// for n_st.  Runs once per determinant set and n_st, on the first FP32 call,
// whose own launch follows.  A stretch of a quarter of the work items (2^18 at
// least) tells the shapes apart: at 3e5, 5e5 and 1e6 determinants with 1, 2, 3,
// 4 and 8 states its fastest shape is the one of all items or within 0.5
// percent of it (65,536 items: within 3 percent).  No shape is the best
// everywhere: loads one trip ahead win with 2 states (0.321 against 0.345 ms at
// 3e5, 2.18 against 2.26 at 1e6) and cost 20 percent with 8.
int tune_sigma32(qpgpu_ctx* c, SigmaItems* it, const SigArgs& all, int nst, cudaStream_t st, int slot) {
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
    cudaGetLastError();
    return qpgpu_fail(c, QPGPU_ERR_CUDA, "cudaEventCreate failed while tuning the FP32 sigma");
  }
  SigArgs a = all;
  const int64_t n = std::min<int64_t>(all.n_items, std::max<int64_t>(all.n_items / 4, 1 << 18));
  const int64_t first = (all.n_items - n) / 2;
  a.n_items = n;
  a.item_row += first;
  a.item_sub += first;
  a.pv += first * nst;
  a.ps += first * nst;
  int best = 0;
  float best_ms = 1e30f;
  for (int v = 0; v < kNSig32Shapes; ++v) {
    launch_any(a, nst, QPGPU_FP32, 1, st, v);
    cudaEventRecord(e0, st);
    launch_any(a, nst, QPGPU_FP32, 1, st, v);
    cudaEventRecord(e1, st);
    if (cudaEventSynchronize(e1) != cudaSuccess) break;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (c->profile) fprintf(stderr, "[qpgpu] sigma32 n_st=%d row=%d floats shape %d: %.3f ms\n", nst, a.u32_ld, v, ms);
    if (ms < best_ms) {
      best_ms = ms;
      best = v;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  QP_CUDA(c, cudaGetLastError());
  it->sig32_variant[slot] = best;
  return 0;
}

}  // namespace

// Work items of the sigma kernels (one per chunk of a row), built after the
// pairs: item starts and the places of the split rows are prefix sums on the
// device (over the host the counts of a 1e6 set took 6.6 ms)
int qp_build_sigma_items(qpgpu_ctx* c, SigmaItems* it) {
  const int64_t N = c->N;
  cudaStream_t st = c->stream;
  it->free_all(c);
  QP_CUDA(c, pool_alloc(c, &it->row_nitems, N + 1));
  QP_CUDA(c, pool_alloc(c, &it->row_item0, N + 1));
  Scoped<int> split(c), split0(c);
  Scoped<char> tmp(c);
  QP_CUDA(c, split.alloc((size_t)N + 1));
  QP_CUDA(c, split0.alloc((size_t)N + 1));
  k_row_nitems<<<gsz(N, 256), 256, 0, st>>>(c->d_rowptr, it->row_nitems, split.p, N);
  size_t tb = 0;
  QP_CUDA(c, cub::DeviceScan::ExclusiveSum(nullptr, tb, it->row_nitems, it->row_item0, (int)(N + 1), st));
  QP_CUDA(c, tmp.alloc(tb));
  QP_CUDA(c, cub::DeviceScan::ExclusiveSum(tmp.p, tb, it->row_nitems, it->row_item0, (int)(N + 1), st));
  QP_CUDA(c, cub::DeviceScan::ExclusiveSum(tmp.p, tb, split.p, split0.p, (int)(N + 1), st));
  int h[2] = {0, 0};
  QP_CUDA(c, cudaMemcpyAsync(&h[0], it->row_item0 + N, sizeof(int), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaMemcpyAsync(&h[1], split0.p + N, sizeof(int), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaStreamSynchronize(st));
  it->n_items = h[0];
  it->n_multi = h[1];
  QP_CUDA(c, pool_alloc(c, &it->item_row, it->n_items));
  QP_CUDA(c, pool_alloc(c, &it->item_sub, it->n_items));
  QP_CUDA(c, pool_alloc(c, &it->multi_rows, (size_t)it->n_multi + 1));
  k_fill_items<<<gsz(N, 256), 256, 0, st>>>(it->row_nitems, it->row_item0, split0.p, it->item_row, it->item_sub,
                                            it->multi_rows, N);
  QP_CUDA(c, cudaGetLastError());
  QP_CUDA(c, cudaStreamSynchronize(st));
  return 0;
}

// Partial-sum buffers sized for nst states.
int qp_ensure_partials(qpgpu_ctx* c, SigmaItems* it, int nst) {
  const size_t need = (size_t)it->n_items * nst;
  if (it->partial_cap >= need) return 0;
  dev_free(c, it->pv);
  dev_free(c, it->ps);
  it->pv = it->ps = nullptr;
  it->partial_cap = 0;
  QP_CUDA(c, dev_alloc(c, &it->pv, need));
  QP_CUDA(c, dev_alloc(c, &it->ps, need));
  it->partial_cap = need;
  return 0;
}

int qp_sigma_launch(qpgpu_ctx* c, SigmaItems* it, double* v, double* s, const double* u, const float* u32, int nst,
                    int precision, cudaStream_t st, int row_lo, int row_hi, int row_first, int row_step,
                    int u32_ld, const float* u32lo) {
  if (nst < 1 || nst > 8) return qpgpu_fail(c, QPGPU_ERR_ARG, "n_st must be in 1..8 per sigma block");
  if (c->direct) return qp_sigma_direct(c, v, s, u, nst, st, row_lo, row_hi, row_first, row_step);
  if (u32_ld <= 0) u32_ld = nst;
  if (u32_ld != nst && !(u32_ld == qp_pad_states(nst) && (((uintptr_t)u32) & 31) == 0))
    return qpgpu_fail(c, QPGPU_ERR_ARG, "FP32 rows must be n_st floats apart, or padded to 4/8 and 32-byte aligned");
  if (precision == QPGPU_FP32 && !u32) return qpgpu_fail(c, QPGPU_ERR_ARG, "FP32 sigma needs u_t32");
  int rc = qp_ensure_partials(c, it, nst);
  if (rc) return rc;
  SigArgs a{};
  a.N = c->N;
  a.rowptr = c->d_rowptr;
  a.colidx = c->d_colidx;
  a.val64 = c->d_val64;
  a.val32 = c->d_val32;
  a.s2ptr = c->d_s2ptr;
  a.s2col = c->d_s2col;
  a.s2val = c->d_s2val;
  a.hdiag = c->d_hdiag;
  a.sdiag = c->d_sdiag;
  a.item_row = it->item_row;
  a.item_sub = it->item_sub;
  a.row_nitems = it->row_nitems;
  a.n_items = it->n_items;
  a.u = u;
  a.u32 = u32;
  a.u32_ld = u32_ld;
  a.u32lo = u32lo;
  a.val32lo = c->d_val32lo;
  if (precision == QPGPU_FF && (!u32lo || !c->d_val32lo || u32_ld != qp_pad_states(nst)))
    return qpgpu_fail(c, QPGPU_ERR_STATE, "float-float sigma needs split coefficients and elements");
  a.v = v;
  a.s = s;
  a.pv = it->pv;
  a.ps = it->ps;
  a.row_lo = row_lo;
  a.row_hi = row_hi;
  a.row_first = row_first;
  a.row_step = row_step;
  const unsigned grid = gsz(it->n_items * 32, SBLK);
  const int slot = nst + (u32_ld != nst ? 9 : 0);
  if (precision == QPGPU_FP32 && it->sig32_variant[slot] < 0) {
    rc = tune_sigma32(c, it, a, nst, st, slot);
    if (rc) return rc;
  }
  launch_any(a, nst, precision, grid, st, it->sig32_variant[slot]);
  if (it->n_multi > 0)
    k_sigma_combine<<<gsz((int64_t)it->n_multi * nst, 256), 256, 0, st>>>(a, it->multi_rows, it->row_item0,
                                                                         it->n_multi, nst);
  QP_CUDA(c, cudaGetLastError());
  return 0;
}

#define QP_PER_NST(nst, CALL)  \
  switch (nst) {               \
    case 1: CALL(1); break;    \
    case 2: CALL(2); break;    \
    case 3: CALL(3); break;    \
    case 4: CALL(4); break;    \
    case 5: CALL(5); break;    \
    case 6: CALL(6); break;    \
    case 7: CALL(7); break;    \
    case 8: CALL(8); break;    \
  }

void qp_to_bilinear(const double* u0, int64_t ld, const int* pos, double* ut, float* ut32, int nst, int64_t N,
                    cudaStream_t st, int* bad) {
#define QP_TO(NS) k_to_bilinear<NS><<<gsz(N, 128), 128, 0, st>>>(u0, ld, pos, ut, ut32, N, bad)
  QP_PER_NST(nst, QP_TO)
#undef QP_TO
}

void qp_flag_nonfinite(const double* x, int64_t n, int* bad, cudaStream_t st) {
  k_nonfinite<<<gsz(n, 256), 256, 0, st>>>(x, n, bad);
}

void qp_from_bilinear(const double* vt, int64_t ld, const int* pos, double* v0, int nst, int64_t N,
                      cudaStream_t st, const double* wt, double* w0) {
#define QP_FROM(NS) k_from_bilinear<NS><<<gsz(N, 128), 128, 0, st>>>(vt, wt, ld, pos, v0, w0, N)
  QP_PER_NST(nst, QP_FROM)
#undef QP_FROM
}

int qp_sigma_ff(qpgpu_ctx* c, SigmaItems* it, double* v, double* s, const double* u, int nst, cudaStream_t st,
                int row_lo, int row_hi, int row_first, int row_step) {
  if (nst < 1 || nst > 8) return qpgpu_fail(c, QPGPU_ERR_ARG, "n_st must be in 1..8 per sigma block");
  if (c->direct) return qp_sigma_direct(c, v, s, u, nst, st, row_lo, row_hi, row_first, row_step);
  const int64_t N = c->N;
  if (!c->d_val32lo) {  // once per determinant set
    QP_CUDA(c, dev_alloc(c, &c->d_val32lo, c->P));
    k_lo_parts<<<gsz(c->P, 256), 256, 0, st>>>(c->d_val64, c->d_val32, c->d_val32lo, c->P);
  }
  const int ld = qp_pad_states(nst);
  const size_t half = ((size_t)N * ld + 63) / 64 * 64;  // keeps lo 256-byte aligned
  if (c->ffu_floats < 2 * half) {
    dev_free(c, c->d_ffu);
    c->d_ffu = nullptr;
    c->ffu_floats = 0;
    QP_CUDA(c, dev_alloc(c, &c->d_ffu, 2 * half));
    c->ffu_floats = 2 * half;
  }
  float* hi = c->d_ffu;
  float* lo = c->d_ffu + half;
  k_split_rows<<<gsz(N * nst, 256), 256, 0, st>>>(u, hi, lo, N, nst, ld);
  return qp_sigma_launch(c, it, v, s, u, hi, nst, QPGPU_FF, st, row_lo, row_hi, row_first, row_step, ld, lo);
}

void qp_to_float(const double* x, float* y, int64_t N, int nst, int ld, cudaStream_t st) {
  k_to_float<<<gsz(N * nst, 256), 256, 0, st>>>(x, y, N, nst, ld);
}

// ---------------------------------------------------------------------------
// Sigma without device allocation.
//
// qpgpu_sigma_bilinear keeps its per-chunk partial sums (rows whose pairs span
// several work chunks) in a buffer that it grows with cudaMalloc on first use.
// Some callers cannot let a library call cudaMalloc: a host code whose device
// memory is owned by its own pool allocator (cudaMalloc fails or fragments the
// pool), or a worker that overlaps sigma with copies and communication on
// other streams, where cudaMalloc/cudaFree would synchronise the device.  For
// them the scratch lives in a fixed device array below, of
// QP_NOALLOC_SLOTS doubles for each of the two sums (8 MiB in total), which
// every GPU that loads this library holds until the process exits.
// ---------------------------------------------------------------------------
#define QP_NOALLOC_SLOTS (1 << 19)
static __device__ __align__(256) double g_noalloc_partials[2 * QP_NOALLOC_SLOTS];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
double* g_noalloc_ptr[kMaxDevices] = {nullptr};  // device address of the array, per device
}  // namespace

extern "C" int qpgpu_sigma_bilinear_noalloc(qpgpu_ctx* c, double* v_t, double* s_t, const double* u_t,
                                            const float* u_t32, int n_st, int precision, void* stream) {
  if (!c) return QPGPU_ERR_ARG;
  if (!c->have_ints || !c->have_pairs) return qpgpu_fail(c, QPGPU_ERR_STATE, "determinants not set");
  if (c->direct) return qpgpu_fail(c, QPGPU_ERR_STATE, "the no-alloc sigma needs stored pairs (direct sigma set)");
  if (!v_t || !s_t || !u_t || n_st < 1 || n_st > 8 || (precision != QPGPU_FP64 && precision != QPGPU_FP32) ||
      (precision == QPGPU_FP32 && !u_t32))
    return qpgpu_fail(c, QPGPU_ERR_ARG, "bad sigma arguments (n_st must be 1..8)");
  if (((uintptr_t)u_t & 15) || (u_t32 && ((uintptr_t)u_t32 & 15)))
    return qpgpu_fail(c, QPGPU_ERR_ARG, "u_t and u_t32 must be 16-byte aligned");
  std::lock_guard<std::mutex> lk(c->mu);
  const SigmaItems* it = &c->items;
  if (it->n_items * (int64_t)n_st > (int64_t)QP_NOALLOC_SLOTS)
    return qpgpu_fail(c, QPGPU_ERR_ARG,
                      "no-alloc sigma: work chunks x n_st exceeds the fixed scratch of 524288 slots");
  // device address of the scratch array on this context's device, looked up
  // once per device (in host code the array's name is not a device address)
  if (c->device < 0 || c->device >= kMaxDevices) return qpgpu_fail(c, QPGPU_ERR_ARG, "device ordinal too large");
  double* scratch = nullptr;
  {
    std::lock_guard<std::mutex> g(g_noalloc_mu);
    if (!g_noalloc_ptr[c->device]) {
      int cur = -1;
      if (cudaGetDevice(&cur) != cudaSuccess) return qpgpu_fail(c, QPGPU_ERR_CUDA, "cudaGetDevice failed");
      if (cur != c->device && cudaSetDevice(c->device) != cudaSuccess)
        return qpgpu_fail(c, QPGPU_ERR_CUDA, "cudaSetDevice failed");
      void* p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partials);
      if (cur != c->device) cudaSetDevice(cur);
      if (e != cudaSuccess) return qpgpu_fail(c, QPGPU_ERR_CUDA, "cudaGetSymbolAddress of the sigma scratch failed");
      g_noalloc_ptr[c->device] = (double*)p;
    }
    scratch = g_noalloc_ptr[c->device];
  }
  SigArgs a{};
  a.N = c->N;
  a.rowptr = c->d_rowptr;
  a.colidx = c->d_colidx;
  a.val64 = c->d_val64;
  a.val32 = c->d_val32;
  a.s2ptr = c->d_s2ptr;
  a.s2col = c->d_s2col;
  a.s2val = c->d_s2val;
  a.hdiag = c->d_hdiag;
  a.sdiag = c->d_sdiag;
  a.item_row = it->item_row;
  a.item_sub = it->item_sub;
  a.row_nitems = it->row_nitems;
  a.n_items = it->n_items;
  a.u = u_t;
  a.u32 = u_t32;
  a.u32_ld = n_st;
  a.v = v_t;
  a.s = s_t;
  a.pv = scratch;  // every slot read by k_sigma_combine is written earlier in the same call
  a.ps = scratch + QP_NOALLOC_SLOTS;
  a.row_lo = 0;
  a.row_hi = (int)c->N;
  a.row_first = 0;
  a.row_step = 1;
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  const unsigned grid = gsz(it->n_items * 32, SBLK);
  launch_any(a, n_st, precision, grid, st, it->sig32_variant[n_st]);
  if (it->n_multi > 0)
    k_sigma_combine<<<gsz((int64_t)it->n_multi * n_st, 256), 256, 0, st>>>(a, it->multi_rows, it->row_item0,
                                                                          it->n_multi, n_st);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return qpgpu_fail(c, QPGPU_ERR_CUDA, cudaGetErrorString(e));
  return QPGPU_OK;
}
