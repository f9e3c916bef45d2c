// Build of the connected-pair Hamiltonian (CSR over bilinear rows).
//
// The pair set is the one H_S2_u_0_nstates_openmp_work visits
// (src/Davidson/u0Hu0.irp.f:177-444): for the determinant I = (a, b) at
// bilinear position k
//   class A  J in the same beta column, alpha strings 1 or 2 apart  (:277-332)
//   class B  J in the same alpha row, beta strings 1 or 2 apart      (:336-415)
//   class C  alpha single x beta single                              (:177-246)
// with the diagonal kept apart (:418-441).
//
// One warp owns a row: it scans the row's beta column (class A), alpha row
// (class B) and the columns of the beta singles of b, or the rows of the alpha
// singles of a, whichever hold fewer determinants (class C); lines with
// deletion-key tables (keys.cu) are probed instead.  Hits are compacted with
// __ballot_sync, so no atomics order them.
//
// Stored pairs.  The scans run once: each warp writes the hits of its rows
// into chunks of a pool and counts them.  k_sort_rows then moves each row's
// hits to their place in the CSR, ascending, and k_pair_values evaluates the
// elements.  At 1e6 determinants the scans take 26 ms (68 ms as a count and a
// fill pass).  Rows that found the pool full are scanned a second time and write
// straight into the CSR; without a pool that is every row.
//
// Direct sigma (sets whose pairs do not fit in device memory).  The scans
// count once at set-up and write one chunk of rows' columns at every sigma
// call, row k's A hits, then its B hits, then its C hits, for k_pair_sigma.
#include <algorithm>
#include <climits>
#include <vector>

#include <cub/cub.cuh>

#include "qpgpu_internal.cuh"
#include "sigma_device.cuh"

namespace {

constexpr int BLK = 256;
constexpr int SAME_BPS = 4, CLASS_C_BPS = 3;  // blocks of the scans resident on an SM, by their registers

inline unsigned nblocks(int64_t n, int tpb) {
  int64_t g = (n + tpb - 1) / tpb;
  return (unsigned)(g < 1 ? 1 : g);
}

struct BuildArgs {
  DevTables t;
  int64_t N;
  const u64* alpha;
  const u64* beta;
  const int* rows;
  const int* cols;
  const int* col_loc;
  const int* t_order;
  const int* row_loc;
  const u64* alpha_pos;  // alpha string at each bilinear position
  const u64* beta_tpos;  // beta string at each alpha-major position
  const int* sa_ptr;
  const int* sa_idx;
  const int* sb_ptr;
  const int* sb_idx;
  const int64_t* cost_a;
  const int64_t* cost_b;
  // hits of each row and class (A, B, C) and spin-flip pairs among the C hits
  int* cnt[3];
  int* cntS;
  // MODE_POOL: pool of columns, handed out in chunks; pos[class][row] = first
  // hit of the row's class in the pool (-1: the pool was full)
  int* pool;
  int64_t pool_cap;
  int pool_chunk[3];
  unsigned long long* pool_next;
  int* pool_full;
  int64_t* pos[3];
  // MODE_POOL: spin-flip pairs (row, place in the row, column, +-1), in any order
  int4* s2rec;
  int64_t s2rec_cap;
  unsigned long long* s2rec_next;
  int write_s2;  // MODE_FILL: write the spin-flip pairs at s2ptr
  unsigned long long* next_row;  // MODE_POOL: rows handed out to warps (one counter per class)
  // CSR (fill pass, sort, elements)
  const int64_t* rowptr;
  int* colidx;
  double* val64;
  float* val32;
  const int64_t* s2ptr;
  int* s2col;
  float* s2val;
  float4* feat;         // .w: coupling strength of the row (learned step)
  // elements and direct sigma: work items (stretches of QP_SIGMA_CHUNK pairs of
  // a row) and, for rows of several, each item's sum of squared elements or its
  // shares of v and s
  const int* row_nitems;
  const int* row_item0;
  const int* item_row;
  const int* item_sub;
  int64_t n_items;
  double* item_sum2;
  double* item_v;
  double* item_s;
  const u64* det_pos;   // both strings at each bilinear position (2 NINT words)
  const u64* det_tpos;  // the same at each alpha-major position (direct sigma)
  int* err;  // set when a fill of the CSR would write past its row's segment (direct sigma: null)
  // direct sigma (k_pair_sigma): v, s = H u, S^2 u for the selected rows, u (N, nst)
  const double* u;
  const double* uT;  // u in alpha-major order: same-alpha partners are contiguous there
  double* v;
  double* s;
  const double* hdiag;
  const double* sdiag;
  int nst;
  // a fill takes the rows row_first modulo row_step of [row_lo, row_hi)
  int row_lo, row_hi, row_first, row_step;
  // chunked direct sigma: the fill writes columns of rows [row_lo, row_hi) at
  // rowptr[k] - col_base, and same-alpha partners are written as alpha-major
  // positions tagged with QP_TAG_T
  int64_t col_base;
  int tag_t;
  // deletion-key tables of the heavy lines (keys.cu); colkey / rowkey null: none
  KeyView kv[KT_N];
  const unsigned char* colkey;
  const unsigned char* rowkey;
  u64 hmask;
};

constexpr unsigned QP_TAG_T = 0x80000000u;  // column given as alpha-major position

constexpr int MODE_COUNT = 0, MODE_FILL = 1, MODE_POOL = 2;
enum { CLS_A = 0, CLS_B = 1, CLS_C = 2 };

__device__ __forceinline__ bool dsel(const BuildArgs& a, int64_t k) {
  return k >= a.row_lo && k < a.row_hi && ((k - a.row_first) % a.row_step) == 0;
}

// Runs `row` on the rows of a scan of one class: MODE_COUNT all rows and
// MODE_FILL the selected ones (with a pool, those that did not fit it) in the
// order of the warps.  MODE_POOL takes them from a counter one at a time, the
// next one while the current one runs: the rows of the lowest excitations
// take up to 0.2 ms each and stand side by side, so that handing out four
// (or 64 a block) left most SMs waiting for the last of them.
template <int MODE, int CLS, class Row>
__device__ __forceinline__ void for_rows(const BuildArgs& a, int lane, Row row) {
  if (MODE == MODE_POOL) {
    unsigned long long next = 0;
    if (lane == 0) next = atomicAdd(a.next_row + CLS, 1ull);
    while (true) {
      const int64_t k = (int64_t)__shfl_sync(0xffffffffu, next, 0);
      if (k >= a.N) return;
      if (lane == 0) next = atomicAdd(a.next_row + CLS, 1ull);
      row(k);
    }
  } else {
    const int64_t step = ((int64_t)gridDim.x * BLK) >> 5;
    const int64_t end = MODE == MODE_FILL ? a.row_hi : a.N;
    const int64_t first = (MODE == MODE_FILL ? a.row_lo : 0) + (int64_t)blockIdx.x * (BLK / 32) + (threadIdx.x >> 5);
#pragma unroll 1
    for (int64_t k = first; k < end; k += step) {
      if (MODE == MODE_FILL && (!dsel(a, k) || (a.pool && a.pos[CLS][k] >= 0))) continue;
      row(k);
    }
  }
}

// Writes the hits of one class of a row after the other.
template <int MODE, int CLS>
struct RowOut {
  int64_t at = 0, keep_at = 0;  // MODE_POOL: this warp's place in the pool and what is left of its chunk,
  int room = 0, keep_room = 0;  // and the largest piece that the row in hand has outgrown
  int* dst = nullptr;
  int cnt = 0, cap = 0;
  __device__ __forceinline__ void begin(const BuildArgs& a, int64_t k) {
    cnt = 0;
    if (MODE == MODE_POOL) {
      dst = a.pool + at;
    } else if (MODE == MODE_FILL) {
      const int before = CLS == CLS_A ? 0 : CLS == CLS_B ? a.cnt[CLS_A][k] : a.cnt[CLS_A][k] + a.cnt[CLS_B][k];
      dst = a.colidx + (a.rowptr[k] - a.col_base + before);
      cap = CLS == CLS_C ? (int)(a.rowptr[k + 1] - a.rowptr[k]) - before : a.cnt[CLS][k];
    }
  }
  // lanes with `hit` append col (every lane calls)
  __device__ __forceinline__ void put(const BuildArgs& a, bool hit, int col, int lane) {
    const unsigned bal = __ballot_sync(0xffffffffu, hit);
    const int n = __popc(bal);
    if (MODE == MODE_POOL && cnt + n > room) grow(a, cnt + n, lane);
    if (MODE != MODE_COUNT && hit) {
      const int o = cnt + __popc(bal & ((1u << lane) - 1u));
      if (MODE == MODE_POOL) {
        if (dst) dst[o] = col;
      } else if (o < cap) {
        dst[o] = col;
      } else if (a.err) {
        atomicOr(a.err, 1 << CLS);
      }
    }
    cnt += n;
  }
  // a new chunk for a row that does not fit the rest of the current one: what
  // the row has so far moves over, and the rows after it go on in the larger
  // of what it leaves (given up, the pieces that the longest rows outgrew and
  // the ends of theirs made the pool of a 1e5 or 2e5 set run full, so that the
  // scans ran again: 0.9 of 7.2 and 1.6 of 13.5 ms)
  __device__ __forceinline__ void grow(const BuildArgs& a, int need, int lane) {
    const int64_t size = min(max((int64_t)a.pool_chunk[CLS], 2 * (int64_t)need), a.N);  // a row holds fewer than N
    unsigned long long o = 0;
    if (lane == 0) o = atomicAdd(a.pool_next, (unsigned long long)size);
    o = __shfl_sync(0xffffffffu, o, 0);
    if (dst == nullptr || (int64_t)o + size > a.pool_cap) {  // full: go on counting
      if (lane == 0) *a.pool_full = 1;
      if (dst) leave();
      dst = nullptr;
      at = 0;
      room = INT_MAX;
      return;
    }
    leave();
    int* to = a.pool + o;
    __syncwarp();
    for (int i0 = 0; i0 < cnt; i0 += 32 * 8) {
      int x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) x[q] = dst[min(i0 + 32 * q + lane, cnt - 1)];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (i0 + 32 * q + lane < cnt) to[i0 + 32 * q + lane] = x[q];
    }
    __syncwarp();
    dst = to;
    at = (int64_t)o;
    room = (int)size;
  }
  __device__ __forceinline__ void leave() {
    if (room > keep_room) {
      keep_at = at;
      keep_room = room;
    }
  }
  __device__ __forceinline__ void end(const BuildArgs& a, int64_t k, int lane) {
    if (MODE == MODE_FILL) return;
    if (lane == 0) a.cnt[CLS][k] = cnt;
    if (MODE == MODE_POOL) {
      if (lane == 0) a.pos[CLS][k] = dst ? at : -1;
      if (dst) {
        at += cnt;
        room -= cnt;
      } else {
        room = 0;
      }
      if (keep_room > room) {
        at = keep_at;
        room = keep_room;
      }
      keep_room = 0;
    }
  }
};

// spin flip test of an alpha-single x beta-single pair: the two excitations
// swap the same two orbitals between the spins (get_s2, s2.irp.f:46-55)
template <int NINT>
__device__ __forceinline__ bool spin_flip(const u64* my, const u64* ca, const u64* cb) {
  bool same = true, core = false;
#pragma unroll
  for (int w = 0; w < NINT; ++w) {
    u64 xa = my[w] ^ ca[w], xb = my[NINT + w] ^ cb[w];
    same &= (xa == xb);
    core |= (xa & my[w] & my[NINT + w]) != 0;
  }
  return same && !core;
}

// ---- class C: alpha single x beta single, one warp per row ----------------
// A column (row) with a 1-deletion table is not scanned: the lanes probe the
// row's alpha (beta) string with each electron removed, and the members of
// each group are the alpha (beta) singles of the row in that column (row).
template <int NINT, int MODE>
__global__ void __launch_bounds__(BLK, CLASS_C_BPS) k_class_c(BuildArgs a) {
  constexpr unsigned FULL = 0xffffffffu;
  // steps of scanned candidates in flight (one: 0.55 instead of 0.42 ms at 1e5
  // determinants, 19.5 instead of 19.2 at 1e6; four need two blocks of an SM: 21.2)
  constexpr int CU = 2;
  const int lane = threadIdx.x & 31;
  RowOut<MODE, CLS_C> out;
  for_rows<MODE, CLS_C>(a, lane, [&](int64_t k) {
    const int ai = a.rows[k], bi = a.cols[k];
    u64 my[2 * NINT];
#pragma unroll
    for (int w = 0; w < NINT; ++w) {
      my[w] = a.alpha[(int64_t)ai * NINT + w];
      my[NINT + w] = a.beta[(int64_t)bi * NINT + w];
    }
    out.begin(a, k);
    int scnt = 0;
    // the spin-flip pairs of a step, in the order of the scan, with <I|S^2|J>
    auto put_flip = [&](bool flip, unsigned fb, const u64* ca, const u64* cb, int col) {
      unsigned long long at = 0;
      if (MODE == MODE_POOL) {
        if (lane == 0) at = atomicAdd(a.s2rec_next, (unsigned long long)__popc(fb));
        at = __shfl_sync(FULL, at, 0);
      }
      if (!flip) return;
      u64 J[2 * NINT], E[2 * NINT];
#pragma unroll
      for (int w = 0; w < NINT; ++w) {
        J[w] = ca[w];
        J[NINT + w] = cb[w];
      }
      det_parity<NINT>(my, E);
      double s2;
      h_double_ab<NINT>(a.t, my, J, E, &s2, nullptr, nullptr);
      const int rank = __popc(fb & ((1u << lane) - 1u));
      if (MODE == MODE_POOL) {
        if ((int64_t)at + rank < a.s2rec_cap) a.s2rec[at + rank] = make_int4((int)k, scnt + rank, col, (int)s2);
      } else if (a.s2ptr[k] + scnt + rank < a.s2ptr[k + 1]) {
        a.s2col[a.s2ptr[k] + scnt + rank] = col;
        a.s2val[a.s2ptr[k] + scnt + rank] = (float)s2;
      } else {
        atomicOr(a.err, 8);
      }
    };
    // 32 candidates, one per lane: hit = (ca, cb) is an alpha single x beta
    // single of the row, written as col
    auto step = [&](bool hit, const u64* ca, const u64* cb, int col) {
      if (MODE != MODE_FILL || a.write_s2) {
        const bool flip = hit && spin_flip<NINT>(my, ca, cb);
        const unsigned fb = __ballot_sync(FULL, flip);
        if (MODE != MODE_COUNT && fb) put_flip(flip, fb, ca, cb, col);
        scnt += __popc(fb);
      }
      out.put(a, hit, col, lane);
    };
    // Lines of the row's singles, 32 at a time: the lanes read the bounds of
    // 32 lines at once, and the candidates of the scanned ones are packed
    // into full warp steps (lane prefix sums over the line lengths), since
    // most lines hold a few determinants; lines with a 1-deletion table are
    // probed afterwards, one after the other.
    const bool by_cols = a.cost_b[bi] <= a.cost_a[ai];
    const int t_beg = by_cols ? a.sb_ptr[bi] : a.sa_ptr[ai];
    const int t_end = by_cols ? a.sb_ptr[bi + 1] : a.sa_ptr[ai + 1];
    const int* lidx = by_cols ? a.sb_idx : a.sa_idx;
    const int* lloc = by_cols ? a.col_loc : a.row_loc;
    const unsigned char* lkey = by_cols ? a.colkey : a.rowkey;
    for (int t0 = t_beg; t0 < t_end; t0 += 32) {
      const int t = t0 + lane;
      int ln = -1, beg = 0, len = 0;
      bool kl = false;
      if (t < t_end) {
        ln = lidx[t];
        beg = lloc[ln];
        kl = lkey && (lkey[ln] & KEY_SINGLE);
        if (!kl) len = lloc[ln + 1] - beg;
      }
      int incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += y;
      }
      const int total = __shfl_sync(FULL, incl, 31);
      for (int c0 = 0; c0 < total; c0 += 32 * CU) {
        int pos[CU], sln[CU];
        u64 y[CU][NINT];  // the scanned strings: alpha of a column, beta of a row
#pragma unroll
        for (int q = 0; q < CU; ++q) {
          const int ci = c0 + 32 * q + lane;
          int src = 0;  // first lane whose inclusive prefix exceeds ci
#pragma unroll
          for (int st = 16; st > 0; st >>= 1) {
            const int pr = __shfl_sync(FULL, incl, src + st - 1);
            if (pr <= ci) src += st;
          }
          const int sbeg = __shfl_sync(FULL, beg, src), slen = __shfl_sync(FULL, len, src);
          const int sinc = __shfl_sync(FULL, incl, src);
          sln[q] = __shfl_sync(FULL, ln, src);
          pos[q] = ci < total ? sbeg + (ci - (sinc - slen)) : -1;
          const u64* const str = (by_cols ? a.alpha_pos : a.beta_tpos) + (int64_t)max(pos[q], 0) * NINT;
#pragma unroll
          for (int w = 0; w < NINT; ++w) y[q][w] = str[w];
        }
#pragma unroll
        for (int q = 0; q < CU; ++q) {
          if (c0 + 32 * q >= total) break;
          int d = 0;
#pragma unroll
          for (int w = 0; w < NINT; ++w) d += popc64((by_cols ? my[w] : my[NINT + w]) ^ y[q][w]);
          // column sln (a beta single): alpha singles of the row; row sln (an
          // alpha single): beta singles of the row
          const bool hit = pos[q] >= 0 && d == 2;
          u64 ca[NINT], cb[NINT];
#pragma unroll
          for (int w = 0; w < NINT; ++w) ca[w] = cb[w] = 0;
          int col = 0;
          if (hit) {
            const u64* const line = (by_cols ? a.beta : a.alpha) + (int64_t)sln[q] * NINT;
#pragma unroll
            for (int w = 0; w < NINT; ++w) {
              const u64 z = line[w];
              ca[w] = by_cols ? y[q][w] : z;
              cb[w] = by_cols ? z : y[q][w];
            }
            if (by_cols)
              col = pos[q];
            else if (MODE != MODE_COUNT)
              col = a.tag_t ? (int)(QP_TAG_T | (unsigned)pos[q]) : a.t_order[pos[q]];
          }
          step(hit, ca, cb, col);
        }
      }
      unsigned kb = __ballot_sync(FULL, kl);
      while (kb) {
        const int L = __ffs(kb) - 1;
        kb &= kb - 1;
        const int kln = __shfl_sync(FULL, ln, L);
        const int kbeg = lloc[kln], kend = lloc[kln + 1];
        // keyed line: the lanes probe the row's string (alpha in a column,
        // beta in a row) minus each electron; the members of a group are its
        // singles in that line
        u64 xs[NINT];  // the row's string of the probed spin
#pragma unroll
        for (int w = 0; w < NINT; ++w) xs[w] = by_cols ? my[w] : my[NINT + w];
        const int ne = by_cols ? a.t.na : a.t.nb;
        const int kind = by_cols ? KT_COL1 : KT_ROW1;
        const KeyView& kv = a.kv[kind];
        u64 fixed[NINT];  // the string of the line's other spin
#pragma unroll
        for (int w = 0; w < NINT; ++w) fixed[w] = by_cols ? a.beta[(int64_t)kln * NINT + w] : a.alpha[(int64_t)kln * NINT + w];
        for (int e0 = 0; e0 < ne; e0 += 32) {
          unsigned gs = 0, gl = 0;
          u64 K[NINT];
#pragma unroll
          for (int w = 0; w < NINT; ++w) K[w] = xs[w];
          if (e0 + lane < ne) {
            const int eb = nth_electron<NINT>(K, e0 + lane);
            clear_orbital<NINT>(K, eb);
            if (!key_find(kv, key_hash<NINT>(kind, kln, K, a.hmask), gs, gl)) gl = 0;
          }
          // the members of the 32 probed groups, packed into full warp steps
          int inc = (int)gl;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, inc, o);
            if (lane >= o) inc += y;
          }
          const int tot = __shfl_sync(FULL, inc, 31);
          for (int m0 = 0; m0 < tot; m0 += 32) {
            const int mi = m0 + lane;
            int src = 0;
#pragma unroll
            for (int st = 16; st > 0; st >>= 1) {
              const int pr = __shfl_sync(FULL, inc, src + st - 1);
              if (pr <= mi) src += st;
            }
            const unsigned s0 = __shfl_sync(FULL, gs, src);
            const int i0 = __shfl_sync(FULL, inc, src) - (int)__shfl_sync(FULL, gl, src);
            u64 Kr[NINT];
#pragma unroll
            for (int w = 0; w < NINT; ++w) Kr[w] = __shfl_sync(FULL, K[w], src);
            {
              int pos = -1;
              if (mi < tot) {
                const unsigned tt = (unsigned)(mi - i0);
                pos = kv.mem[s0 + tt];
                if (tt > 0 && kv.mem[s0 + tt - 1] == pos) pos = -1;  // repeated member (colliding keys)
              }
              bool hit = false;
              u64 ca[NINT], cb[NINT];
#pragma unroll
              for (int w = 0; w < NINT; ++w) ca[w] = cb[w] = 0;
              int col = 0;
              if (pos >= kbeg && pos < kend) {
                int d = 0;
                bool eq = true;
                u64 y[NINT];
#pragma unroll
                for (int w = 0; w < NINT; ++w) {
                  y[w] = by_cols ? a.alpha_pos[(int64_t)pos * NINT + w] : a.beta_tpos[(int64_t)pos * NINT + w];
                  d += popc64(xs[w] ^ y[w]);
                  eq &= (xs[w] & y[w]) == Kr[w];
                }
                hit = d == 2 && eq;
                if (hit) {
#pragma unroll
                  for (int w = 0; w < NINT; ++w) {
                    ca[w] = by_cols ? y[w] : fixed[w];
                    cb[w] = by_cols ? fixed[w] : y[w];
                  }
                  if (by_cols)
                    col = pos;
                  else if (MODE != MODE_COUNT)
                    col = a.tag_t ? (int)(QP_TAG_T | (unsigned)pos) : a.t_order[pos];
                }
              }
              step(hit, ca, cb, col);
            }
          }
        }
      }
    }
    out.end(a, k, lane);
    if (MODE != MODE_FILL && lane == 0) a.cntS[k] = scnt;
  });
}

// ---- same-spin pairs, one warp per row -------------------------------------
// SPIN 0: the row's beta column (class A), SPIN 1: its alpha row (class B).
// A line without a 2-deletion table is scanned, 32 strings a step.  In a line
// with one the lanes probe 32 of the row's C(ne,2) keys at a time; then the
// members of the 32 groups are packed into full warp steps (most groups hold
// a few strings).
// A member y of the key K of x is a double when |x ^ y| = 4 and x & y = K,
// and a single when |x ^ y| = 2 and K is x & y without its lowest electron:
// each pair is accepted under exactly one key, whatever the hash collisions.
// (A thread per row of a line staged in shared memory took 140 us for each
// fill of a 5,000 determinant set, whose longest line gave 20 blocks work.)
// A group of 64 members or more is read by itself, four steps in flight and
// without the search for each member's group: the reference's row, one warp
// whose groups are that long, bounds the scan (5.0 and 5.4 of 5.0 and 5.4 ms
// at 1e6 determinants, now 3.6 and 4.0; 1.10 and 1.17 -> 0.80 and 0.71 at 2e5).
// Groups from 32 or 128 on made no difference; registers for five blocks of an
// SM spill (3.9 and 4.6 ms).
template <int NINT, int MODE, int SPIN>
__global__ void __launch_bounds__(BLK, SAME_BPS) k_same(BuildArgs a) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int GU = 4;  // steps of a large group in flight
  constexpr int kind = SPIN == 0 ? KT_COL2 : KT_ROW2;
  const int lane = threadIdx.x & 31;
  const KeyView kv = a.kv[kind];
  const int ne = SPIN == 0 ? a.t.na : a.t.nb;
  const int nc = ne * (ne - 1) / 2;
  const unsigned char* lflag = SPIN == 0 ? a.colkey : a.rowkey;
  const u64* strs = SPIN == 0 ? a.alpha_pos : a.beta_tpos;
  constexpr int CLS = SPIN == 0 ? CLS_A : CLS_B;
  RowOut<MODE, CLS> out;
  for_rows<MODE, CLS>(a, lane, [&](int64_t k) {
    const int line = SPIN == 0 ? a.cols[k] : a.rows[k];
    u64 x[NINT];
#pragma unroll
    for (int w = 0; w < NINT; ++w)
      x[w] = SPIN == 0 ? a.alpha_pos[k * NINT + w] : a.beta[(int64_t)a.cols[k] * NINT + w];
    const int ls = SPIN == 0 ? a.col_loc[line] : a.row_loc[line];
    const int le = SPIN == 0 ? a.col_loc[line + 1] : a.row_loc[line + 1];
    out.begin(a, k);
    auto column = [&](int p) {
      return MODE == MODE_COUNT || SPIN == 0 ? p : (a.tag_t ? (int)(QP_TAG_T | (unsigned)p) : a.t_order[p]);
    };
    if (!(lflag && (lflag[line] & KEY_DOUBLE))) {
      for (int p0 = ls; p0 < le; p0 += 32) {
        const int p = p0 + lane;
        bool hit = false;
        if (p < le) {
          int d = 0;
#pragma unroll
          for (int w = 0; w < NINT; ++w) d += popc64(x[w] ^ strs[(int64_t)p * NINT + w]);
          hit = d == 2 || d == 4;
        }
        out.put(a, hit, hit ? column(p) : 0, lane);
      }
      out.end(a, k, lane);
      return;
    }
    // the string at p is a partner of the row under key Kr
    auto partner = [&](int p, const u64 (&Kr)[NINT]) {
      u64 m[NINT];
      int d = 0;
#pragma unroll
      for (int w = 0; w < NINT; ++w) {
        const u64 y = strs[(int64_t)p * NINT + w];
        d += popc64(x[w] ^ y);
        m[w] = x[w] & y;
      }
      if (d == 2) {  // canonical key of a single: drop the lowest common electron
        bool done = false;
#pragma unroll
        for (int w = 0; w < NINT; ++w)
          if (!done && m[w]) {
            m[w] &= m[w] - 1;
            done = true;
          }
      }
      bool eq = d == 2 || d == 4;
#pragma unroll
      for (int w = 0; w < NINT; ++w) eq &= m[w] == Kr[w];
      return eq;
    };
    for (int c0 = 0; c0 < nc; c0 += 32) {
      unsigned gs = 0, gl = 0;
      u64 K[NINT];
#pragma unroll
      for (int w = 0; w < NINT; ++w) K[w] = 0;
      if (c0 + lane < nc) {
        int i, j;
        pair_of_combo(c0 + lane, ne, i, j);
        const int bi = nth_electron<NINT>(x, i), bj = nth_electron<NINT>(x, j);
#pragma unroll
        for (int w = 0; w < NINT; ++w) K[w] = x[w];
        clear_orbital<NINT>(K, bi);
        clear_orbital<NINT>(K, bj);
        if (!key_find(kv, key_hash<NINT>(kind, line, K, a.hmask), gs, gl)) gl = 0;
      }
      // groups of two warp steps or more, one after the other: GU x 32 members
      // a trip, whose loads are in flight together
      unsigned large = __ballot_sync(FULL, gl >= 64);
      while (large) {
        const int L = __ffs(large) - 1;
        large &= large - 1;
        const int* mem = kv.mem + __shfl_sync(FULL, gs, L);
        const int len = (int)__shfl_sync(FULL, gl, L);
        u64 Kr[NINT];
#pragma unroll
        for (int w = 0; w < NINT; ++w) Kr[w] = __shfl_sync(FULL, K[w], L);
        if (lane == L) gl = 0;
        for (int t0 = 0; t0 < len; t0 += 32 * GU) {
          int p[GU];
          bool hit[GU];
#pragma unroll
          for (int q = 0; q < GU; ++q) {
            const int t = t0 + 32 * q + lane;
            p[q] = t < len ? mem[t] : -1;
            if (t > 0 && t < len && mem[t - 1] == p[q]) p[q] = -1;  // repeated member
          }
#pragma unroll
          for (int q = 0; q < GU; ++q) hit[q] = p[q] >= ls && p[q] < le && partner(p[q], Kr);
#pragma unroll
          for (int q = 0; q < GU; ++q) p[q] = hit[q] ? column(p[q]) : 0;
#pragma unroll
          for (int q = 0; q < GU; ++q)
            if (t0 + 32 * q < len) out.put(a, hit[q], p[q], lane);
        }
      }
      // the members of the other groups, packed into full warp steps
      int inc = (int)gl;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += y;
      }
      const int tot = __shfl_sync(FULL, inc, 31);
      for (int m0 = 0; m0 < tot; m0 += 32) {
        const int mi = m0 + lane;
        int src = 0;
#pragma unroll
        for (int st = 16; st > 0; st >>= 1) {
          const int pr = __shfl_sync(FULL, inc, src + st - 1);
          if (pr <= mi) src += st;
        }
        const unsigned s0 = __shfl_sync(FULL, gs, src);
        const int i0 = __shfl_sync(FULL, inc, src) - (int)__shfl_sync(FULL, gl, src);
        u64 Kr[NINT];
#pragma unroll
        for (int w = 0; w < NINT; ++w) Kr[w] = __shfl_sync(FULL, K[w], src);
        const unsigned t = (unsigned)(mi - i0);
        bool hit = false;
        int p = 0;
        if (mi < tot) {
          p = kv.mem[s0 + t];
          const bool dup = t > 0 && kv.mem[s0 + t - 1] == p;
          hit = !dup && p >= ls && p < le && partner(p, Kr);
        }
        out.put(a, hit, hit ? column(p) : 0, lane);
      }
    }
    out.end(a, k, lane);
  });
}

// ---- each row's columns, ascending -----------------------------------------
// Neighbouring lanes of the sigma gathers then read neighbouring coefficients,
// whatever order the scans found the partners in.  Bitonic networks in
// registers: element i of a row sits in register i % R of lane i / R, so of
// the 55 steps of 1,024 elements 40 run inside a thread, 15 across lanes and
// none needs shared memory; rows of 1,025 to 16,384 elements add exchanges between
// up to 16 such warps through shared memory, longer ones go to a segmented
// radix sort.  991M columns at 1e6 determinants: 10.2 ms (7.2 of them in the
// rows of 2,049 to 4,096), against 43.2 ms for a segmented sort of every row.
constexpr int SORT_WARP = 1024;          // elements of a warp
constexpr int SORT_PAD = SORT_WARP + SORT_WARP / 32;

// ascending merge of each thread's R registers (a bitonic run), steps J, J/2, ..., 1
template <int R, int J = R / 2>
__device__ __forceinline__ void merge_regs(unsigned (&v)[R]) {
  if constexpr (J > 0) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if ((r & J) == 0) {
        const unsigned lo = min(v[r], v[r | J]), hi = max(v[r], v[r | J]);
        v[r] = lo;
        v[r | J] = hi;
      }
    merge_regs<R, J / 2>(v);
  }
}
// runs of K < R registers, their directions alternating (compile-time steps:
// an array indexed by a loop variable would go to local memory)
template <int R, int K, int J>
__device__ __forceinline__ void short_runs(unsigned (&v)[R]) {
#pragma unroll
  for (int r = 0; r < R; ++r)
    if ((r & J) == 0) {
      const unsigned lo = min(v[r], v[r | J]), hi = max(v[r], v[r | J]);
      v[r] = (r & K) == 0 ? lo : hi;
      v[r | J] = (r & K) == 0 ? hi : lo;
    }
  if constexpr (J > 1) short_runs<R, K, J / 2>(v);
  else if constexpr (2 * K < R) short_runs<R, 2 * K, K>(v);
}
template <int R>
__device__ __forceinline__ void flip(unsigned (&v)[R], unsigned m) {
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] ^= m;
}
// A bitonic run of `lanes` lanes, ascending: strides over lanes, then inside a
// thread.  The loops stay loops: the network written out is 56 KB of
// instructions, which the warps of an SM then fetch at different places.
template <int R>
__device__ __forceinline__ void merge_lanes(unsigned (&v)[R], int lane, int lanes) {
#pragma unroll 1
  for (int j = lanes / 2; j > 0; j >>= 1) {
    const bool low = (lane & j) == 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const unsigned o = __shfl_xor_sync(0xffffffffu, v[r], j);
      v[r] = low ? min(v[r], o) : max(v[r], o);
    }
  }
  merge_regs<R>(v);
}
// The 32 R elements of a warp (element i in register i % R of lane i / R),
// ascending when `up`.  A descending run is an ascending one of the
// complements, so only the signs of the values change with the direction.
template <int R>
__device__ __forceinline__ void sort_warp(unsigned (&v)[R], int lane, bool up) {
  if constexpr (R > 2) short_runs<R, 2, 1>(v);
  unsigned m = 0;
#pragma unroll 1
  for (int lanes = 1; lanes <= 32; lanes <<= 1) {
    const unsigned want = (lanes == 32 ? up : (lane & lanes) == 0) ? 0u : 0xffffffffu;
    flip<R>(v, m ^ want);
    m = want;
    merge_lanes<R>(v, lane, lanes);
  }
  flip<R>(v, m);
}
// a bitonic sequence of 32 R elements, ascending when `up`
template <int R>
__device__ __forceinline__ void merge_warp(unsigned (&v)[R], int lane, bool up) {
  const unsigned m = up ? 0u : 0xffffffffu;
  flip<R>(v, m);
  merge_lanes<R>(v, lane, 32);
  flip<R>(v, m);
}

// hit i of row k: from the pool (classes one after the other) or its place in the CSR
struct RowSrc {
  const int* src[3];
  int n0 = INT_MAX, n1 = INT_MAX;
  __device__ __forceinline__ RowSrc(const BuildArgs& a, int64_t k) {
    src[0] = src[1] = src[2] = a.colidx + a.rowptr[k];
    if (a.pool) {
      n0 = a.cnt[CLS_A][k];
      n1 = n0 + a.cnt[CLS_B][k];
      const int64_t p0 = a.pos[CLS_A][k], p1 = a.pos[CLS_B][k], p2 = a.pos[CLS_C][k];
      if (p0 >= 0) src[0] = a.pool + p0;
      if (p1 >= 0) src[1] = a.pool + p1 - n0;
      if (p2 >= 0) src[2] = a.pool + p2 - n1;
    }
  }
  __device__ __forceinline__ unsigned at(int i) const {
    const int* p = i < n0 ? src[0] : i < n1 ? src[1] : src[2];
    return (unsigned)p[i];
  }
};

template <int R>
__device__ __forceinline__ void sort_row_small(const RowSrc& row, int* out, int n, int lane, unsigned* sm) {
  unsigned v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = r * 32 + lane < n ? row.at(r * 32 + lane) : 0xffffffffu;
  sort_warp<R>(v, lane, true);
  if constexpr (R == 1) {
    if (lane < n) out[lane] = (int)v[0];
  } else {
    // element lane R + r -> coalesced writes (one pad word in 32 keeps the banks apart)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = lane * R + r;
      sm[i + (i >> 5)] = v[r];
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = r * 32 + lane;
      if (i < n) out[i] = (int)sm[i + (i >> 5)];
    }
    __syncwarp();
  }
}

__global__ void __launch_bounds__(BLK, 3) k_sort_rows(BuildArgs a) {
  __shared__ unsigned sm[BLK / 32][SORT_PAD];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t warp = ((int64_t)blockIdx.x * BLK + threadIdx.x) >> 5;
  const int64_t nwarp = ((int64_t)gridDim.x * BLK) >> 5;
  for (int64_t k = warp; k < a.N; k += nwarp) {
    const int64_t e0 = a.rowptr[k], n64 = a.rowptr[k + 1] - e0;
    if (n64 == 0 || n64 > SORT_WARP) continue;
    const int n = (int)n64;
    const RowSrc row(a, k);
    int* out = a.colidx + e0;
    if (n <= 32)
      sort_row_small<1>(row, out, n, lane, sm[w]);
    else if (n <= 128)
      sort_row_small<4>(row, out, n, lane, sm[w]);
    else if (n <= 256)
      sort_row_small<8>(row, out, n, lane, sm[w]);
    else if (n <= 512)
      sort_row_small<16>(row, out, n, lane, sm[w]);
    else
      sort_row_small<32>(row, out, n, lane, sm[w]);
  }
}

// rows of more than 512 W and at most 1024 W columns, a block of W warps each;
// the rows (in any order) and their number come from k_long_rows
template <int W>
__global__ void __launch_bounds__(W * 32, W <= 8 ? 24 / W : 1) k_sort_rows_block(BuildArgs a, const int* list, const int* n_list) {
  extern __shared__ unsigned smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nl = *n_list;
  for (int q = blockIdx.x; q < nl; q += gridDim.x) {
    const int64_t k = list[q];
    const int64_t e0 = a.rowptr[k];
    const int n = (int)(a.rowptr[k + 1] - e0);
    const RowSrc row(a, k);
    unsigned v[32];
#pragma unroll
    for (int r = 0; r < 32; ++r) {
      const int i = w * SORT_WARP + r * 32 + lane;
      v[r] = i < n ? row.at(i) : 0xffffffffu;
    }
    sort_warp<32>(v, lane, (w & 1) == 0);
#pragma unroll 1
    for (int kw = 2; kw <= W; kw <<= 1) {  // runs of kw warps
      const bool up = (w & kw) == 0;
#pragma unroll 1
      for (int jw = kw / 2; jw > 0; jw >>= 1) {
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 32; ++r) smem[w * SORT_PAD + r * 32 + lane] = v[r];
        __syncthreads();
        const bool low = ((w & jw) == 0) == up;
#pragma unroll
        for (int r = 0; r < 32; ++r) {
          const unsigned o = smem[(w ^ jw) * SORT_PAD + r * 32 + lane];
          v[r] = low ? min(v[r], o) : max(v[r], o);
        }
      }
      merge_warp<32>(v, lane, up);
    }
    __syncthreads();
    unsigned* sw = smem + w * SORT_PAD;
#pragma unroll
    for (int r = 0; r < 32; ++r) sw[lane * 33 + r] = v[r];
    __syncwarp();
    int* out = a.colidx + e0;
#pragma unroll
    for (int r = 0; r < 32; ++r) {
      const int i = r * 32 + lane;
      if (w * SORT_WARP + i < n) out[w * SORT_WARP + i] = (int)sw[i + (i >> 5)];
    }
    __syncthreads();
  }
}

// rows longer than SORT_WARP, by the block that sorts them: list[b cap + ...],
// b = 0..3 for 2, 4, 8, 16 warps, b = 4 for the segmented sort, whose rows'
// lengths follow at list[5 cap + ...]
constexpr int SORT_BINS = 5;
__global__ void k_long_rows(const int64_t* rowptr, int64_t N, int64_t cap, int* list, int* n) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < N; k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t len = rowptr[k + 1] - rowptr[k];
    if (len <= SORT_WARP) continue;
    int b = 0;
    while (b < SORT_BINS - 1 && len > (int64_t)SORT_WARP * (2 << b)) ++b;
    const int o = atomicAdd(&n[b], 1);
    if (o >= cap) continue;
    list[b * cap + o] = (int)k;
    if (b == SORT_BINS - 1) list[SORT_BINS * cap + o] = (int)len;
  }
}

// the columns of listed rows, one block per row: into tmp at off[q], or back
__global__ void k_gather_rows(BuildArgs a, const int* list, const int* off, int nl, int* tmp) {
  for (int q = blockIdx.x; q < nl; q += gridDim.x) {
    const RowSrc row(a, list[q]);
    const int n = off[q + 1] - off[q];
    for (int i = threadIdx.x; i < n; i += blockDim.x) tmp[off[q] + i] = (int)row.at(i);
  }
}
__global__ void k_scatter_rows(BuildArgs a, const int* list, const int* off, int nl, const int* tmp) {
  for (int q = blockIdx.x; q < nl; q += gridDim.x) {
    int* out = a.colidx + a.rowptr[list[q]];
    const int n = off[q + 1] - off[q];
    for (int i = threadIdx.x; i < n; i += blockDim.x) out[i] = tmp[off[q] + i];
  }
}

// A warp's list of pairs put off until 32 of them are there (shared memory):
// the rare, long branches of an element kernel then run with all lanes busy.
constexpr int DEFER = 64;
struct Deferred {
  int* q;  // DEFER entries of this warp
  int n;
  // lanes with `on` append x; true when 32 or more are waiting
  __device__ __forceinline__ bool push(bool on, int x, unsigned lt) {
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (on) q[n + __popc(m & lt)] = x;
    n += __popc(m);
    __syncwarp();
    return n >= 32;
  }
  // the last up to 32 entries, one per lane (-1: none)
  __device__ __forceinline__ int pop(int lane) {
    const int m = min(n, 32);
    n -= m;
    const int x = lane < m ? q[n + lane] : -1;
    __syncwarp();
    return x;
  }
};

// both strings of a determinant in one load (det_pos / det_tpos: 16 or 32 bytes a row)
template <int NINT>
__device__ __forceinline__ void load_det(const u64* det, int64_t p, u64 (&J)[2 * NINT]) {
  if constexpr (NINT == 1) {
    const ulonglong2 x = __ldg(reinterpret_cast<const ulonglong2*>(det) + p);
    J[0] = x.x;
    J[1] = x.y;
  } else {
    asm("ld.global.nc.v4.u64 {%0,%1,%2,%3}, [%4];"
        : "=l"(J[0]), "=l"(J[1]), "=l"(J[2]), "=l"(J[3])
        : "l"(det + p * 4));
  }
}

// FP64 / FP32 elements of the stored pairs, after their columns are in place:
// one warp per row, lanes over the row's pairs, so that the integral loads of
// 32 pairs are in flight at once.  A partner's two strings sit in one 32-byte
// sector (det_pos): with the strings behind the beta id, a pair took four
// requests and a chain of three dependent loads before its integral.  Each
// class calls the same Slater routine with the same arguments as the scans
// do, so the values are bit-identical.  Single excitations (whose sums over
// the holes and particles against the reference take several times a double's
// loads), and same-spin doubles where they are few in a trip, are deferred
// until 32 of a kind are there (a row's own beta column is one run of its
// ascending columns, whose trips take them at once).  The row's sum of squared
// elements gives the coupling feature of the learned step
// (log10(sum_J H_IJ^2) / 4), which took a pass of its own (4.2 ms).
// A warp takes a stretch of QP_SIGMA_CHUNK pairs: with a warp per row the
// reference's row, which holds up to a quarter of the determinants, ran on
// when the others were done.  The next trip's partners are loaded ahead, for
// which three blocks of an SM have registers (four without: 20.8 ms at 1e6).
// 1e5 (60 MOs) / 2e5 / 1e6 determinants: 1.26 / 3.0 / 21.3 -> 0.70 / 1.75 /
// 19.1 ms; bound by the Slater routines (about 400 integer instructions a pair,
// 42 percent issue, FP64 pipe at 62) with the L2 latency of the integrals.
__device__ __forceinline__ float coupling_feature(double sum2) { return (float)(log10(sum2 + 1e-30) * 0.25); }

template <int NINT>
__global__ void __launch_bounds__(BLK, 3) k_pair_values(BuildArgs a) {
  __shared__ int s_q[BLK / 32][2][DEFER];
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t warp = ((int64_t)blockIdx.x * BLK + threadIdx.x) >> 5;
  const int64_t nwarp = ((int64_t)gridDim.x * BLK) >> 5;
  Deferred same{s_q[threadIdx.x >> 5][0], 0}, mono{s_q[threadIdx.x >> 5][1], 0};
  for (int64_t it = warp; it < a.n_items; it += nwarp) {
    const int k = a.item_row[it];
    u64 my[2 * NINT], E[2 * NINT];
    load_det<NINT>(a.det_pos, k, my);
    det_parity<NINT>(my, E);
    const int64_t e0 = a.rowptr[k] + (int64_t)a.item_sub[it] * QP_SIGMA_CHUNK;
    const int n = (int)min((int64_t)QP_SIGMA_CHUNK, a.rowptr[k + 1] - e0);
    double sum2 = 0.0;
    auto put = [&](int x, double v) {
      a.val64[e0 + x] = v;
      a.val32[e0 + x] = (float)v;
      sum2 = fma(v, v, sum2);
    };
    auto do_mono = [&](int x) {  // one string differs, by one electron
      if (x < 0) return;
      u64 J[2 * NINT];
      load_det<NINT>(a.det_pos, a.colidx[e0 + x], J);
      bool beta = true;
#pragma unroll
      for (int w = 0; w < NINT; ++w) beta &= my[w] == J[w];
      put(x, h_mono_spin<NINT>(a.t, my, J, E, beta ? 2 : 1, nullptr, nullptr));
    };
    auto same_spin = [&](int x, const u64 (&J)[2 * NINT]) -> bool {  // true: a single
      bool beta = true;
      int d = 0;
#pragma unroll
      for (int w = 0; w < NINT; ++w) beta &= my[w] == J[w];
      u64 si[NINT], sj[NINT], Es[NINT];
#pragma unroll
      for (int w = 0; w < NINT; ++w) {
        si[w] = beta ? my[NINT + w] : my[w];
        sj[w] = beta ? J[NINT + w] : J[w];
        Es[w] = beta ? E[NINT + w] : E[w];
        d += popc64(si[w] ^ sj[w]);
      }
      if (d == 2) return true;
      put(x, h_double_spin<NINT>(a.t, si, sj, Es, nullptr, nullptr));
      return false;
    };
    auto do_same = [&](int x) -> bool {
      if (x < 0) return false;
      u64 J[2 * NINT];
      load_det<NINT>(a.det_pos, a.colidx[e0 + x], J);
      return same_spin(x, J);
    };
    int j = lane < n ? a.colidx[e0 + lane] : -1;
    int jn = lane + 32 < n ? a.colidx[e0 + lane + 32] : -1;
    u64 Jn[2 * NINT];
#pragma unroll
    for (int w = 0; w < 2 * NINT; ++w) Jn[w] = 0;
    if (j >= 0) load_det<NINT>(a.det_pos, j, Jn);
    for (int x0 = 0; x0 < n; x0 += 32) {
      const int x = x0 + lane;
      const int jnn = x + 64 < n ? a.colidx[e0 + x + 64] : -1;  // two trips ahead
      bool is_same = false;
      u64 J[2 * NINT];
#pragma unroll
      for (int w = 0; w < 2 * NINT; ++w) J[w] = Jn[w];
      if (jn >= 0) load_det<NINT>(a.det_pos, jn, Jn);
      if (j >= 0) {
        bool samea = true, sameb = true;
#pragma unroll
        for (int w = 0; w < NINT; ++w) {
          samea &= J[w] == my[w];
          sameb &= J[NINT + w] == my[NINT + w];
        }
        is_same = samea || sameb;
        double s2;
        if (!is_same) put(x, h_double_ab<NINT>(a.t, my, J, E, &s2, nullptr, nullptr));
      }
      if (__popc(__ballot_sync(0xffffffffu, is_same)) >= 12) {
        if (mono.push(is_same && same_spin(x, J), x, lt)) do_mono(mono.pop(lane));
      } else if (same.push(is_same, x, lt)) {
        const int y = same.pop(lane);
        if (mono.push(do_same(y), y, lt)) do_mono(mono.pop(lane));
      }
      j = jn;
      jn = jnn;
    }
    {
      const int y = same.pop(lane);
      if (mono.push(do_same(y), y, lt)) do_mono(mono.pop(lane));
    }
    do_mono(mono.pop(lane));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum2 += __shfl_xor_sync(0xffffffffu, sum2, o);
    if (lane == 0) {
      if (a.row_nitems[k] == 1)
        a.feat[k].w = coupling_feature(sum2);
      else
        a.item_sum2[it] = sum2;
    }
  }
}

// the coupling feature of the rows of several items: their sums in item order
__global__ void k_row_coupling(BuildArgs a, const int* multi_rows, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int k = multi_rows[i];
    double s = 0.0;
    for (int j = 0; j < a.row_nitems[k]; ++j) s += a.item_sum2[a.row_item0[k] + j];
    a.feat[k].w = coupling_feature(s);
  }
}

// out[p] = strings of the determinant at bilinear position p (perm null) or at
// alpha-major position p (perm = t_order)
template <int NINT>
__global__ void k_det_pos(const u64* alpha, const u64* beta, const int* rows, const int* cols, const int* perm,
                          u64* out, int64_t N) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < N; p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = perm ? perm[p] : p;
#pragma unroll
    for (int w = 0; w < NINT; ++w) {
      out[p * 2 * NINT + w] = alpha[(int64_t)rows[k] * NINT + w];
      out[p * 2 * NINT + NINT + w] = beta[(int64_t)cols[k] * NINT + w];
    }
  }
}

// the recorded spin-flip pairs to their places
__global__ void k_s2_scatter(const int4* rec, int64_t n, const int64_t* s2ptr, int* s2col, float* s2val) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int4 r = rec[i];
    s2col[s2ptr[r.x] + r.y] = r.z;
    s2val[s2ptr[r.x] + r.y] = (float)r.w;
  }
}

__global__ void k_row_totals(const int* A, const int* B, const int* C, const int* S, int64_t* tot, int64_t* stot,
                             int64_t N) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k <= N; k += (int64_t)gridDim.x * blockDim.x) {
    tot[k] = (k < N) ? (int64_t)A[k] + B[k] + C[k] : 0;
    stot[k] = (k < N) ? (int64_t)S[k] : 0;
  }
}

// H_II and <I|S+S-|I> in bilinear order (diag_H_mat_elem, slater_rules.irp.f:1869;
// diag_S_mat_elem, s2.irp.f:1-30)
template <int NINT>
__global__ void k_diag(DevTables t, const u64* alpha, const u64* beta, const int* rows, const int* cols,
                       double* hd, double* sd, float* hd32, int64_t N) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < N; k += (int64_t)gridDim.x * blockDim.x) {
    u64 det[2 * NINT];
    const int ai = rows[k], bi = cols[k];
#pragma unroll
    for (int w = 0; w < NINT; ++w) {
      det[w] = alpha[(int64_t)ai * NINT + w];
      det[NINT + w] = beta[(int64_t)bi * NINT + w];
    }
    const double h = diag_h<NINT>(t, det);
    hd[k] = h;
    hd32[k] = (float)h;
    sd[k] = diag_s<NINT>(det);
  }
}

BuildArgs index_args(const qpgpu_ctx* c) {
  BuildArgs a{};
  a.t = c->tab;
  a.N = c->N;
  a.alpha = c->d_alpha;
  a.beta = c->d_beta;
  a.rows = c->d_rows;
  a.cols = c->d_cols;
  a.col_loc = c->d_col_loc;
  a.t_order = c->d_t_order;
  a.row_loc = c->d_row_loc;
  a.alpha_pos = c->d_alpha_pos;
  a.beta_tpos = c->d_beta_tpos;
  a.sa_ptr = c->d_sa_ptr;
  a.sa_idx = c->d_sa_idx;
  a.sb_ptr = c->d_sb_ptr;
  a.sb_idx = c->d_sb_idx;
  a.cost_a = c->d_cost_a;
  a.cost_b = c->d_cost_b;
  a.row_lo = 0;
  a.row_hi = (int)c->N;
  a.row_first = 0;
  a.row_step = 1;
  a.col_base = 0;
  a.tag_t = 0;
  for (int t = 0; t < KT_N; ++t) {
    a.kv[t].slot = c->d_kslot[t];
    a.kv[t].mask = c->kslots[t] > 0 ? (u64)(c->kslots[t] - 1) : 0ull;
    a.kv[t].mem = c->d_kmem[t];
  }
  a.colkey = c->d_colkey;
  a.rowkey = c->d_rowkey;
  a.hmask = c->key_mask;
  return a;
}

template <int W>
int sort_block_bin(qpgpu_ctx* c, const BuildArgs& a, const int* list, const int* n_list, int n) {
  if (n == 0) return 0;
  const int smem = W * SORT_PAD * (int)sizeof(unsigned);
  if (smem > 48 * 1024)
    QP_CUDA(c, cudaFuncSetAttribute(k_sort_rows_block<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  k_sort_rows_block<W><<<(unsigned)std::min(n, c->n_sm * 64), W * 32, smem, c->stream>>>(a, list, n_list);
  return 0;
}

// every row's columns to their place in the CSR, ascending (from the pool, or
// in place when a.pool is null)
int sort_row_columns(qpgpu_ctx* c, const BuildArgs& a) {
  const int64_t N = c->N;
  cudaStream_t st = c->stream;
  if (c->P == 0) return 0;
  k_sort_rows<<<nblocks(N * 32, BLK), BLK, 0, st>>>(a);
  // at most P / 1025 rows are longer than a warp's share
  const int64_t cap = std::min<int64_t>(N, c->P / (SORT_WARP + 1));
  if (cap == 0) return 0;
  Scoped<int> list(c), num(c);
  QP_CUDA(c, list.alloc((size_t)(SORT_BINS + 1) * cap));
  QP_CUDA(c, num.alloc(SORT_BINS));
  QP_CUDA(c, cudaMemsetAsync(num.p, 0, SORT_BINS * sizeof(int), st));
  k_long_rows<<<std::min(nblocks(N, 256), (unsigned)c->n_sm * 8), 256, 0, st>>>(c->d_rowptr, N, cap, list.p, num.p);
  int hn[SORT_BINS];
  QP_CUDA(c, cudaMemcpyAsync(hn, num.p, sizeof(hn), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaStreamSynchronize(st));
  int rc = sort_block_bin<2>(c, a, list.p, num.p, hn[0]);
  if (!rc) rc = sort_block_bin<4>(c, a, list.p + cap, num.p + 1, hn[1]);
  if (!rc) rc = sort_block_bin<8>(c, a, list.p + 2 * cap, num.p + 2, hn[2]);
  if (!rc) rc = sort_block_bin<16>(c, a, list.p + 3 * cap, num.p + 3, hn[3]);
  if (rc) return rc;
  QP_CUDA(c, cudaGetLastError());
  if (hn[4] == 0) return 0;
  // the few rows beyond a block: gathered into one buffer, at most 2^28
  // columns (or one row) at a time, sorted as segments and written back
  const int* lrow = list.p + 4 * cap;
  std::vector<int> len(hn[4]);
  QP_CUDA(c, cudaMemcpyAsync(len.data(), lrow + cap, len.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaStreamSynchronize(st));
  for (size_t q0 = 0; q0 < len.size();) {
    std::vector<int> off{0};
    size_t q1 = q0;
    int64_t sum = 0;
    while (q1 < len.size() && (q1 == q0 || sum + len[q1] <= ((int64_t)1 << 28))) {
      sum += len[q1++];
      if (sum >= ((int64_t)1 << 31) - 1) return qpgpu_fail(c, QPGPU_ERR_NOMEM, "a row holds more than 2^31 pairs");
      off.push_back((int)sum);
    }
    const int nl = (int)(q1 - q0);
    Scoped<int> doff(c), t0(c), t1(c);
    Scoped<char> work(c);
    QP_CUDA(c, doff.alloc(off.size()));
    QP_CUDA(c, t0.alloc((size_t)sum));
    QP_CUDA(c, t1.alloc((size_t)sum));
    QP_CUDA(c, cudaMemcpyAsync(doff.p, off.data(), off.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    k_gather_rows<<<(unsigned)std::min(nl, 65535), 512, 0, st>>>(a, lrow + q0, doff.p, nl, t0.p);
    size_t tb = 0;
    QP_CUDA(c, cub::DeviceSegmentedSort::SortKeys(nullptr, tb, t0.p, t1.p, (int)sum, nl, doff.p, doff.p + 1, st));
    QP_CUDA(c, work.alloc(tb));
    QP_CUDA(c, cub::DeviceSegmentedSort::SortKeys(work.p, tb, t0.p, t1.p, (int)sum, nl, doff.p, doff.p + 1, st));
    k_scatter_rows<<<(unsigned)std::min(nl, 65535), 512, 0, st>>>(a, lrow + q0, doff.p, nl, t1.p);
    QP_CUDA(c, cudaGetLastError());
    QP_CUDA(c, cudaStreamSynchronize(st));  // off is read by the copy
    q0 = q1;
  }
  return 0;
}

// The scans of all three classes, side by side: each of them ends with the
// reference's row in one warp (0.8, 0.7 and 1.1 ms at 2e5 determinants, where
// the other rows keep the device busy for 0.3, 0.3 and 1.0).  A whole set-up
// takes 6.2 ms side by side and 6.8 one after the other at 1e5 determinants,
// 3.54 and 3.69 at 32,768, 2.31 and 2.34 at 5,000: below the line the gain is
// under 0.15 ms, and a context that holds only small sets has no streams.
constexpr int64_t SIDE_BY_SIDE = 1 << 15;
template <int NINT, int MODE>
int launch_scans(qpgpu_ctx* c, const BuildArgs& a, unsigned gs, unsigned gc, cudaStream_t st) {
  const bool side = c->N >= SIDE_BY_SIDE;
  int rc = side ? qp_fork(c, st) : 0;
  if (rc) return rc;
  k_same<NINT, MODE, 0><<<gs, BLK, 0, st>>>(a);
  k_same<NINT, MODE, 1><<<gs, BLK, 0, side ? c->side[0] : st>>>(a);
  k_class_c<NINT, MODE><<<gc, BLK, 0, side ? c->side[1] : st>>>(a);
  rc = side ? qp_join(c, st) : 0;
  if (rc) {  // work arrays are given back on c->stream
    cudaStreamSynchronize(c->side[0]);
    cudaStreamSynchronize(c->side[1]);
  }
  return rc;
}

// the scans of a set-up; a pool pass runs as many blocks as are resident
template <int NINT, int MODE>
int setup_scans(qpgpu_ctx* c, const BuildArgs& a) {
  const unsigned g = nblocks(c->N * 32, BLK);
  const unsigned gs = MODE == MODE_POOL ? std::min(g, (unsigned)c->n_sm * SAME_BPS) : g;
  const unsigned gc = MODE == MODE_POOL ? std::min(g, (unsigned)c->n_sm * CLASS_C_BPS) : g;
  const int rc = launch_scans<NINT, MODE>(c, a, gs, gc, c->stream);
  qp_mark(c, "pair scans");
  return rc;
}

template <int NINT>
int build_pairs_t(qpgpu_ctx* c) {
  const int64_t N = c->N;
  cudaStream_t st = c->stream;
  BuildArgs a = index_args(c);
  Scoped<int> cA(c), cB(c), cC(c), cS(c), pool(c);
  Scoped<int4> s2rec(c);
  Scoped<int64_t> pos(c);
  Scoped<unsigned long long> ctr(c);
  QP_CUDA(c, cA.alloc(N));
  QP_CUDA(c, cB.alloc(N));
  QP_CUDA(c, cC.alloc(N));
  QP_CUDA(c, cS.alloc(N));
  // next row of each class; next free entry of the pool; its full flag; next spin-flip record
  QP_CUDA(c, ctr.alloc(8));
  QP_CUDA(c, cudaMemsetAsync(ctr.p, 0, 8 * sizeof(unsigned long long), st));
  a.cnt[CLS_A] = cA.p;
  a.cnt[CLS_B] = cB.p;
  a.cnt[CLS_C] = cC.p;
  a.cntS = cS.p;
  a.next_row = ctr.p;
  a.pool_next = ctr.p + 3;
  a.pool_full = (int*)(ctr.p + 4);
  a.s2rec_next = ctr.p + 5;
  qp_mark(c, "pair setup");
  size_t fr = 0, total = 0;
  QP_CUDA(c, qp_free_bytes(c, &fr, &total));
  if (c->sigma_mode != QPGPU_SIGMA_DIRECT) {
    // room for as many pairs a row as the context's last set had (1,200 when
    // it had none; the bench system has 991 at 1e6 determinants), 0.3 of that
    // for what rows leave behind when they outgrow a chunk, and for the
    // unfinished chunks of the warps; a pool that is too small costs its rows a
    // second scan, one that would not fit beside the stored pairs is left out
    // (or given up, once their number is known)
    const double per_row = c->pairs_per_row > 0 ? c->pairs_per_row : 1200.0;
    const double est = per_row * (double)N;
    // chunks: an eighth of a warp's share of about 0.3 / 0.3 / 0.6 of the
    // pairs, but sixteen rows at least, as a row that does not fit the rest of
    // a chunk takes another (of 300 pairs in a new context: with 1,200 the
    // chunks of a 5,000 determinant set took 300 MB, 0.3 of 2.5 ms to map), and
    // a row's most at most: the 3 N^2 entries that bound the pool are then a
    // chunk of each class for every row (a 900 determinant set, whose warps have
    // a row each, found it full and was scanned twice)
    const double usual = c->pairs_per_row > 0 ? per_row : 300.0;
    const int64_t all = nblocks(N * 32, BLK);
    const int64_t ws = std::min<int64_t>(all, c->n_sm * SAME_BPS) * (BLK / 32);
    const int64_t wc = std::min<int64_t>(all, c->n_sm * CLASS_C_BPS) * (BLK / 32);
    auto chunk_of = [&](double share, int64_t warps) {
      return (int)std::min({65536.0, (double)N,
                            std::max({256.0, share * est / (8.0 * (double)warps), 16.0 * share * usual})});
    };
    a.pool_chunk[CLS_A] = a.pool_chunk[CLS_B] = chunk_of(0.3, ws);
    a.pool_chunk[CLS_C] = chunk_of(0.6, wc);
    const double slack = 2.0 * (double)ws * a.pool_chunk[CLS_A] + (double)wc * a.pool_chunk[CLS_C];
    const double cap = std::min(1.3 * est + slack, 3.0 * (double)N * (double)N);
    const bool room = 16.0 * est + 4.0 * cap + 28.0 * (double)N + (double)total / 16.0 < (double)fr;
    a.s2rec_cap = 4 * N + (1 << 16);
    if (room && pool.alloc((size_t)cap + 1) == cudaSuccess && pos.alloc(3 * (size_t)N) == cudaSuccess &&
        s2rec.alloc((size_t)a.s2rec_cap) == cudaSuccess) {
      a.s2rec = s2rec.p;
      a.pool = pool.p;
      a.pool_cap = (int64_t)cap;
      for (int q = 0; q < 3; ++q) a.pos[q] = pos.p + q * N;
    } else {
      cudaGetLastError();
      pool.reset();
      pos.reset();
      s2rec.reset();
    }
  }
  const int rcs = a.pool ? setup_scans<NINT, MODE_POOL>(c, a) : setup_scans<NINT, MODE_COUNT>(c, a);
  if (rcs) return rcs;
  QP_CUDA(c, cudaGetLastError());
  Scoped<int64_t> tot(c), stot(c);
  QP_CUDA(c, tot.alloc(N + 1));
  QP_CUDA(c, stot.alloc(N + 1));
  k_row_totals<<<nblocks(N + 1, 256), 256, 0, st>>>(cA.p, cB.p, cC.p, cS.p, tot.p, stot.p, N);
  QP_CUDA(c, pool_alloc(c, &c->d_rowptr, N + 1));
  QP_CUDA(c, pool_alloc(c, &c->d_s2ptr, N + 1));
  size_t tb = 0;
  QP_CUDA(c, cub::DeviceScan::ExclusiveSum(nullptr, tb, tot.p, c->d_rowptr, (int)(N + 1), st));
  Scoped<char> tmp(c);
  QP_CUDA(c, tmp.alloc(tb));
  QP_CUDA(c, cub::DeviceScan::ExclusiveSum(tmp.p, tb, tot.p, c->d_rowptr, (int)(N + 1), st));
  QP_CUDA(c, cub::DeviceScan::ExclusiveSum(tmp.p, tb, stot.p, c->d_s2ptr, (int)(N + 1), st));
  int full = 0;
  QP_CUDA(c, cudaMemcpyAsync(&c->P, c->d_rowptr + N, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaMemcpyAsync(&c->P_s2, c->d_s2ptr + N, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaMemcpyAsync(&full, a.pool_full, sizeof(int), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaStreamSynchronize(st));
  const int64_t P = c->P, PS = c->P_s2;
  c->pairs_per_row = (double)P / (double)N;
  // stored pairs (16 B each, S^2 pairs 8 B) or the direct sigma: forced by
  // qpgpu_set_sigma_mode, else direct when the stored pairs would leave less
  // than 1/16 of the device memory free
  const double need = 16.0 * (double)P + 8.0 * (double)PS + 28.0 * (double)N, margin = (double)total / 16.0;
  bool direct = c->sigma_mode == QPGPU_SIGMA_DIRECT;
  if (c->sigma_mode == QPGPU_SIGMA_AUTO) direct = need + margin > (double)fr;
  c->direct = direct;
  // a set with more pairs than the pool was sized for may fit the device, but
  // not beside the pool: its rows are then scanned a second time
  const double hits = 4.0 * (double)a.pool_cap + 24.0 * (double)N + 16.0 * (double)a.s2rec_cap;
  if (a.pool && (direct || need + margin + hits > (double)fr)) {
    pool.reset();
    pos.reset();
    s2rec.reset();
    a.pool = nullptr;
  }
  if (a.pool && PS > a.s2rec_cap) {  // not all spin-flip pairs recorded: class C again, for every row
    QP_CUDA(c, cudaMemsetAsync(a.pos[CLS_C], 0xff, (size_t)N * sizeof(int64_t), st));
    full = 1;
    a.write_s2 = 1;
  }
  if (!a.pool) a.write_s2 = 1;
  QP_CUDA(c, pool_alloc(c, &c->d_hdiag, N));
  QP_CUDA(c, pool_alloc(c, &c->d_sdiag, N));
  QP_CUDA(c, pool_alloc(c, &c->d_hdiag32, N));
  k_diag<NINT><<<nblocks(N, 256), 256, 0, st>>>(c->tab, c->d_alpha, c->d_beta, c->d_rows, c->d_cols, c->d_hdiag,
                                                 c->d_sdiag, c->d_hdiag32, N);
  qp_mark(c, "row starts, diagonal");
  Scoped<u64> det(c);
  QP_CUDA(c, det.alloc(2 * NINT * (size_t)N));
  k_det_pos<NINT><<<nblocks(N, 256), 256, 0, st>>>(c->d_alpha, c->d_beta, c->d_rows, c->d_cols, nullptr, det.p, N);
  if (direct) {
    // the direct sigma regenerates the columns chunk by chunk: keep the
    // per-row counts of the same-spin classes and the row starts on the host
    c->d_cntA = cA.p;
    cA.p = nullptr;
    c->d_cntB = cB.p;
    cB.p = nullptr;
    c->d_det_pos = det.p;
    det.p = nullptr;
    QP_CUDA(c, pool_alloc(c, &c->d_det_tpos, 2 * NINT * (size_t)N));
    k_det_pos<NINT><<<nblocks(N, 256), 256, 0, st>>>(c->d_alpha, c->d_beta, c->d_rows, c->d_cols, c->d_t_order,
                                                      c->d_det_tpos, N);
    c->h_rowptr.resize(N + 1);
    QP_CUDA(c, cudaMemcpyAsync(c->h_rowptr.data(), c->d_rowptr, (N + 1) * sizeof(int64_t), cudaMemcpyDeviceToHost,
                               st));
    QP_CUDA(c, cudaGetLastError());
    return qp_build_sigma_items(c, &c->items);  // waits for the stream
  }
  if (pool_alloc(c, &c->d_colidx, P) != cudaSuccess || pool_alloc(c, &c->d_val64, P) != cudaSuccess ||
      pool_alloc(c, &c->d_val32, P) != cudaSuccess || pool_alloc(c, &c->d_s2col, PS) != cudaSuccess ||
      pool_alloc(c, &c->d_s2val, PS) != cudaSuccess || pool_alloc(c, &c->d_detfeat, (size_t)N * 4) != cudaSuccess) {
    cudaGetLastError();
    return qpgpu_fail(c, QPGPU_ERR_NOMEM,
                      "not enough device memory for " + std::to_string(P) + " connected pairs");
  }
  a.rowptr = c->d_rowptr;
  a.colidx = c->d_colidx;
  a.val64 = c->d_val64;
  a.val32 = c->d_val32;
  a.s2ptr = c->d_s2ptr;
  a.s2col = c->d_s2col;
  a.s2val = c->d_s2val;
  a.det_pos = det.p;
  a.feat = (float4*)c->d_detfeat;
  Scoped<int> err(c);
  QP_CUDA(c, err.alloc(1));
  QP_CUDA(c, cudaMemsetAsync(err.p, 0, sizeof(int), st));
  a.err = err.p;
  if (!a.pool || full) {
    const int rcf = setup_scans<NINT, MODE_FILL>(c, a);
    if (rcf) return rcf;
    int herr = 0;
    QP_CUDA(c, cudaMemcpyAsync(&herr, err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    QP_CUDA(c, cudaStreamSynchronize(st));
    if (herr)
      return qpgpu_fail(c, QPGPU_ERR_STATE, "pair fill disagrees with pair count (" + std::to_string(herr) + ")");
  }
  if (!a.write_s2 && PS > 0)
    k_s2_scatter<<<nblocks(PS, 256), 256, 0, st>>>(a.s2rec, PS, c->d_s2ptr, c->d_s2col, c->d_s2val);
  const int rc = sort_row_columns(c, a);
  if (rc) return rc;
  qp_mark(c, "row columns sorted");
  pool.reset();
  const int rci = qp_build_sigma_items(c, &c->items);
  if (rci) return rci;
  qp_mark(c, "sigma work items");
  Scoped<double> sum2(c);
  QP_CUDA(c, sum2.alloc((size_t)c->items.n_items));
  a.row_nitems = c->items.row_nitems;
  a.row_item0 = c->items.row_item0;
  a.item_row = c->items.item_row;
  a.item_sub = c->items.item_sub;
  a.n_items = c->items.n_items;
  a.item_sum2 = sum2.p;
  k_pair_values<NINT><<<nblocks(a.n_items * 32, BLK), BLK, 0, st>>>(a);
  if (c->items.n_multi > 0)
    k_row_coupling<<<nblocks(c->items.n_multi, 256), 256, 0, st>>>(a, c->items.multi_rows, c->items.n_multi);
  qp_mark(c, "pair elements");
  QP_CUDA(c, cudaGetLastError());
  int herr = 0;
  QP_CUDA(c, cudaMemcpyAsync(&herr, err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaStreamSynchronize(st));
  if (herr) return qpgpu_fail(c, QPGPU_ERR_STATE, "pair fill disagrees with pair count (" + std::to_string(herr) + ")");
  return 0;
}

__global__ void k_alpha_major(const double* u, const int* t_order, double* uT, int64_t N, int nst) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < N * nst; t += (int64_t)gridDim.x * blockDim.x)
    uT[t] = u[(int64_t)t_order[t / nst] * nst + t % nst];
}

// Direct sigma of the rows [row_lo, row_hi) of one chunk, after the fill
// scans wrote their columns into pc (at rowptr[k] - col_base): one warp per
// stretch of a row, lanes over its pairs; each pair's element is evaluated as in
// k_pair_values (same routines, same arguments), multiplied by the partner's
// coefficients (same-alpha partners, tagged with their alpha-major position,
// read from the alpha-major copy uT, where a row's partners are contiguous),
// and the lanes are combined in a fixed order (as are the stretches of a row,
// k_direct_combine).  The fill wrote the row's
// same-beta partners, then its same-alpha partners, then the alpha x beta
// ones, so each class has a loop of its own, a same-spin partner reads only
// the string it does not share with the row, and the single excitations of
// both same-spin classes are deferred until 32 are there (k_pair_values).
// NP: states padded to a power of two, so that the sums stay in registers.
// 2e5 determinants in 120 MOs, 2 states: 7.4 -> 4.1 ms with the register-only
// Slater routines, the loops per class and the deferred singles; about 1.8
// since a warp takes a stretch of QP_SIGMA_CHUNK pairs and not a row (the
// reference's row outlasted the others; the whole sigma 6.9 -> 4.6 ms, 4.0 with the scans side by side).
template <int NINT, int NP>
__global__ void __launch_bounds__(BLK, 3) k_pair_sigma(BuildArgs a, const int* __restrict__ pc) {
  __shared__ int s_q[BLK / 32][DEFER];
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t warp = ((int64_t)blockIdx.x * BLK + threadIdx.x) >> 5;
  const int64_t nwarp = ((int64_t)gridDim.x * BLK) >> 5;
  const int nst = a.nst;
  Deferred mono{s_q[threadIdx.x >> 5], 0};
  const int64_t it_end = a.row_item0[a.row_hi];
  for (int64_t it = a.row_item0[a.row_lo] + warp; it < it_end; it += nwarp) {
    const int64_t k = a.item_row[it];
    if (((k - a.row_first) % a.row_step) != 0) continue;
    u64 my[2 * NINT], E[2 * NINT];
    const int bi = a.cols[k];
#pragma unroll
    for (int w = 0; w < NINT; ++w) {
      my[w] = a.alpha_pos[k * NINT + w];
      my[NINT + w] = a.beta[(int64_t)bi * NINT + w];
    }
    det_parity<NINT>(my, E);
    double acc[NP], sacc[NP];
#pragma unroll
    for (int st = 0; st < NP; ++st) acc[st] = sacc[st] = 0.0;
    auto add = [&](double (&s)[NP], double v, const double* uj) {
#pragma unroll
      for (int st = 0; st < NP; ++st)
        if (st < nst) s[st] = fma(v, __ldg(uj + st), s[st]);
    };
    const int first = a.item_sub[it] * QP_SIGMA_CHUNK;
    const int64_t e0 = a.rowptr[k] + first;
    const int* prow = pc + (e0 - a.col_base);
    const int n = (int)min((int64_t)QP_SIGMA_CHUNK, a.rowptr[k + 1] - e0);
    const int ra = a.cnt[CLS_A][k] - first;  // where the classes of the row end in this stretch
    const int nA = min(max(ra, 0), n), nB = min(max(ra + a.cnt[CLS_B][k], 0), n);
    auto do_mono = [&](int x) {
      if (x < 0) return;
      const bool beta = x >= nA;
      const int q = (int)((unsigned)prow[x] & ~QP_TAG_T);
      const u64* str = beta ? a.beta_tpos : a.alpha_pos;
      u64 J[2 * NINT];
#pragma unroll
      for (int w = 0; w < NINT; ++w) {
        const u64 y = str[(int64_t)q * NINT + w];
        J[w] = beta ? my[w] : y;
        J[NINT + w] = beta ? y : my[NINT + w];
      }
      const double v = h_mono_spin<NINT>(a.t, my, J, E, beta ? 2 : 1, nullptr, nullptr);
      add(acc, v, (beta ? a.uT : a.u) + (int64_t)q * nst);
    };
    for (int x0 = 0; x0 < nB; x0 += 32) {  // same-spin partners (beta column, then alpha row)
      const int x = x0 + lane;
      bool is_mono = false;
      if (x < nB) {
        const bool beta = x >= nA;
        const int q = (int)((unsigned)prow[x] & ~QP_TAG_T);
        const u64* str = beta ? a.beta_tpos : a.alpha_pos;
        u64 I[NINT], J[NINT], Es[NINT];
        int d = 0;
#pragma unroll
        for (int w = 0; w < NINT; ++w) {
          J[w] = str[(int64_t)q * NINT + w];
          I[w] = beta ? my[NINT + w] : my[w];
          Es[w] = beta ? E[NINT + w] : E[w];
          d += popc64(I[w] ^ J[w]);
        }
        is_mono = d == 2;
        if (!is_mono)
          add(acc, h_double_spin<NINT>(a.t, I, J, Es, nullptr, nullptr), (beta ? a.uT : a.u) + (int64_t)q * nst);
      }
      if (mono.push(is_mono, x, lt)) do_mono(mono.pop(lane));
    }
    for (int x = nB + lane; x < n; x += 32) {  // alpha single x beta single
      const unsigned cj = (unsigned)prow[x];
      const bool via_t = (cj & QP_TAG_T) != 0;
      const int q = (int)(cj & ~QP_TAG_T);
      u64 J[2 * NINT];
      load_det<NINT>(via_t ? a.det_tpos : a.det_pos, q, J);
      double s2;
      const double v = h_double_ab<NINT>(a.t, my, J, E, &s2, nullptr, nullptr);
      const double* uj = (via_t ? a.uT : a.u) + (int64_t)q * nst;
      add(acc, v, uj);
      if (s2 != 0.0) add(sacc, s2, uj);
    }
    __syncwarp();
    do_mono(mono.pop(lane));
    constexpr int SH = 5 - qpsig::Pow2<NP>::lg;
    const double hv = qpsig::reduce_scatter64<NP>(acc, lane);
    const double sv = qpsig::reduce_scatter64<NP>(sacc, lane);
    const int st = lane >> SH;
    if ((lane & ((1 << SH) - 1)) == 0 && st < nst) {
      if (a.row_nitems[k] > 1) {
        a.item_v[it * nst + st] = hv;
        a.item_s[it * nst + st] = sv;
      } else {
        const double uk = a.u[k * nst + st];
        a.v[k * nst + st] = hv + a.hdiag[k] * uk;
        a.s[k * nst + st] = sv + a.sdiag[k] * uk;
      }
    }
  }
}

// the rows of several stretches: their shares in order, then the diagonal
__global__ void k_direct_combine(BuildArgs a, const int* multi_rows, int n) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n * a.nst; t += gridDim.x * blockDim.x) {
    const int64_t k = multi_rows[t / a.nst];
    const int st = t % a.nst;
    if (!dsel(a, k)) continue;
    double hv = 0.0, sv = 0.0;
    for (int j = 0; j < a.row_nitems[k]; ++j) {
      const int64_t it = a.row_item0[k] + j;
      hv += a.item_v[it * a.nst + st];
      sv += a.item_s[it * a.nst + st];
    }
    const double uk = a.u[k * a.nst + st];
    a.v[k * a.nst + st] = hv + a.hdiag[k] * uk;
    a.s[k * a.nst + st] = sv + a.sdiag[k] * uk;
  }
}

template <int NINT>
void launch_pair_sigma(const BuildArgs& a, const int* pc, unsigned grid, cudaStream_t st) {
  switch (qp_pad_states(a.nst)) {
    case 1: k_pair_sigma<NINT, 1><<<grid, BLK, 0, st>>>(a, pc); break;
    case 2: k_pair_sigma<NINT, 2><<<grid, BLK, 0, st>>>(a, pc); break;
    case 4: k_pair_sigma<NINT, 4><<<grid, BLK, 0, st>>>(a, pc); break;
    default: k_pair_sigma<NINT, 8><<<grid, BLK, 0, st>>>(a, pc); break;
  }
}

// chunks of rows whose columns fit the buffer: fill scans restricted to the
// chunk (S^2 lists not written), then k_pair_sigma
template <int NINT>
int sigma_direct_t(qpgpu_ctx* c, double* v, double* s, const double* u, const double* uT, int nst,
                   cudaStream_t st, int row_lo, int row_hi, int row_first, int row_step) {
  BuildArgs a = index_args(c);
  a.u = u;
  a.uT = uT;
  a.v = v;
  a.s = s;
  a.hdiag = c->d_hdiag;
  a.sdiag = c->d_sdiag;
  a.nst = nst;
  a.rowptr = c->d_rowptr;
  a.s2ptr = c->d_s2ptr;
  a.cnt[CLS_A] = c->d_cntA;
  a.cnt[CLS_B] = c->d_cntB;
  a.det_pos = c->d_det_pos;
  a.det_tpos = c->d_det_tpos;
  a.colidx = c->d_direct_cols;
  a.tag_t = 1;
  a.row_first = row_first;
  a.row_step = row_step;
  const int rci = qp_ensure_partials(c, &c->items, nst);
  if (rci) return rci;
  a.row_nitems = c->items.row_nitems;
  a.row_item0 = c->items.row_item0;
  a.item_row = c->items.item_row;
  a.item_sub = c->items.item_sub;
  a.item_v = c->items.pv;
  a.item_s = c->items.ps;
  const int64_t N = c->N;
  const std::vector<int64_t>& rp = c->h_rowptr;
  int64_t clo = 0;
  while (clo < N) {
    // largest chi with rp[chi] - rp[clo] <= capacity (at least one row)
    const int64_t lim = rp[clo] + c->direct_cols_cap;
    int64_t chi = std::upper_bound(rp.begin() + clo + 1, rp.end(), lim) - rp.begin() - 1;
    if (chi <= clo) chi = clo + 1;
    const int64_t lo = std::max<int64_t>(clo, row_lo), hi = std::min<int64_t>(chi, row_hi);
    if (lo < hi) {
      a.row_lo = (int)lo;
      a.row_hi = (int)hi;
      a.col_base = rp[lo];
      const unsigned gK = nblocks((hi - lo) * 32, BLK);
      const bool marks = st == c->stream;  // QPGPU_PROFILE=1: phase times on the context stream
      if (marks) qp_mark(c, "direct: chunk start");
      const int rcs = launch_scans<NINT, MODE_FILL>(c, a, gK, gK, st);
      if (rcs) return rcs;
      if (marks) qp_mark(c, "direct: scans");
      const int64_t items = hi - lo + (rp[hi] - rp[lo]) / QP_SIGMA_CHUNK;  // at most
      launch_pair_sigma<NINT>(a, c->d_direct_cols, nblocks(items * 32, BLK), st);
      if (c->items.n_multi > 0)
        k_direct_combine<<<nblocks((int64_t)c->items.n_multi * nst, 256), 256, 0, st>>>(a, c->items.multi_rows,
                                                                                       c->items.n_multi);
      if (marks) qp_mark(c, "direct: elements");
    }
    clo = chi;
  }
  QP_CUDA(c, cudaGetLastError());
  return 0;
}

}  // namespace

// Direct sigma (FP64, nothing stored): v, s of the rows selected by (row_lo,
// row_hi, row_first, row_step), bilinear order, u (N, nst).
int qp_sigma_direct(qpgpu_ctx* c, double* v, double* s, const double* u, int nst, cudaStream_t st, int row_lo,
                    int row_hi, int row_first, int row_step) {
  if (nst < 1 || nst > 8) return qpgpu_fail(c, QPGPU_ERR_ARG, "n_st must be in 1..8 per sigma block");
  if (row_step < 1) return qpgpu_fail(c, QPGPU_ERR_ARG, "row step must be >= 1");
  const size_t need = (size_t)c->N * nst;
  if (c->direct_ut_n < need) {
    dev_free(c, c->d_direct_ut);
    c->d_direct_ut = nullptr;
    c->direct_ut_n = 0;
    QP_CUDA(c, dev_alloc(c, &c->d_direct_ut, need));
    c->direct_ut_n = need;
  }
  if (!c->d_direct_cols) {  // column buffer: the whole set if it fits in half the free memory
    size_t fr = 0, total = 0;
    QP_CUDA(c, qp_free_bytes(c, &fr, &total));
    int64_t maxrow = 0;
    for (int64_t k = 0; k < c->N; ++k) maxrow = std::max(maxrow, c->h_rowptr[k + 1] - c->h_rowptr[k]);
    int64_t cap = std::min<int64_t>(c->P, (int64_t)(fr / 2 / sizeof(int)));
    // QPGPU_DIRECT_CHUNK_COLS caps the buffer (a memory budget; small values
    // force many chunks)
    if (const char* e = getenv("QPGPU_DIRECT_CHUNK_COLS")) cap = std::min<int64_t>(cap, atoll(e) > 0 ? atoll(e) : cap);
    cap = std::max<int64_t>(cap, maxrow);
    QP_CUDA(c, dev_alloc(c, &c->d_direct_cols, (size_t)std::max<int64_t>(cap, 1)));
    c->direct_cols_cap = cap;
  }
  k_alpha_major<<<nblocks((int64_t)need, 256), 256, 0, st>>>(u, c->d_t_order, c->d_direct_ut, c->N, nst);
  const int rc = (c->nint == 1)
                     ? sigma_direct_t<1>(c, v, s, u, c->d_direct_ut, nst, st, row_lo, row_hi, row_first, row_step)
                     : sigma_direct_t<2>(c, v, s, u, c->d_direct_ut, nst, st, row_lo, row_hi, row_first, row_step);
  if (rc) return rc;
  QP_CUDA(c, cudaGetLastError());
  qp_report_marks(c);
  return 0;
}

void qp_free_pairs(qpgpu_ctx* c) {
  void** ps[] = {(void**)&c->d_rowptr, (void**)&c->d_colidx, (void**)&c->d_val64, (void**)&c->d_val32,
                 (void**)&c->d_s2ptr, (void**)&c->d_s2col, (void**)&c->d_s2val, (void**)&c->d_hdiag,
                 (void**)&c->d_sdiag, (void**)&c->d_hdiag32};
  for (auto p : ps) {
    qp_pool_free(c, *p);
    *p = nullptr;
  }
  c->have_pairs = false;
  c->direct = false;
  void** dp[] = {(void**)&c->d_cntA, (void**)&c->d_cntB, (void**)&c->d_det_pos, (void**)&c->d_det_tpos};
  for (auto p : dp) {
    qp_pool_free(c, *p);
    *p = nullptr;
  }
  // grown by a sigma on the caller's stream: not from the pool
  void** up[] = {(void**)&c->d_val32lo, (void**)&c->d_direct_cols};
  for (auto p : up) {
    dev_free(c, *p);
    *p = nullptr;
  }
  c->direct_cols_cap = 0;
  c->h_rowptr.clear();
  c->P = c->P_s2 = 0;
}

int qp_build_pairs(qpgpu_ctx* c) {
  if (c->nint == 1) return build_pairs_t<1>(c);
  if (c->nint == 2) return build_pairs_t<2>(c);
  return qpgpu_fail(c, QPGPU_ERR_ARG, "n_int > 2 is not supported");
}
