// CIPSI selection with the Epstein-Nesbet second-order energy on the device
// (plugins/Full_CI_ZMQ/selection.irp.f: select_connected :24-79, the
// per-generator walk :258-580, splash_pq and get_d0/d1/d2 :647-1086, the
// banned masks :1088-1172, fill_buffer_double :582-645, and the buffer of
// selection_buffer.irp.f:33-138).
//
// The wave function held by the context must be in psi_det_sorted order:
// generators are determinants 0..n_gen-1 and selectors 0..n_sel-1.
//
// Work items.  For a generator g, an external determinant a is a single
// excitation (g minus a hole h, plus a particle p) or a double one (g minus
// holes h1, h2, plus particles p1, p2).  The particles are orbitals empty in
// g, so each a has exactly one (holes, particles) description.  One CTA
// takes one item (g, holes, range of particle entries):
//  * single: entries p over the empty orbitals of the hole's spin;
//  * same-spin double: entries p1 < p2 over the empty orbitals of the
//    holes' spin;
//  * alpha-beta double: entries (p1 alpha, p2 beta).
// The entry range of an item is cut so that its numerator tile (entries x
// states, FP64) fits the CTA's shared memory.
//
// Numerators.  mask = g without the holes.  A selector D can be connected
// (excitation degree <= 2) to some a = mask + particles only if D lacks at
// most two of mask's electrons (k = |mask \ D| <= 2).  For a double item,
// a and D are then connected iff k + [p1 not in D] + [p2 not in D] <= 2; for
// a single item, iff k + [p not in D] <= 2.  This is the case split of
// get_d0 / get_d1 / get_d2 with k = 0, 1, 2.  Only selectors within a
// quadruple excitation of g can pass, so those are listed once per
// generator (k_sel_lists).  The CTA filters them per item (k <= 2), in
// selector order.  Every thread owns a fixed set of entries and adds
// c_D <a|H|D> for its connected entries, selector after selector, so each
// numerator is summed in selector order with no atomics.  <a|H|D> is the
// generic i_H_j (slater_rules.irp.f:478-570) with a as the first
// determinant.
//
// Few of the staged selectors are connected to an entry, so the tile is also
// kept transposed: one bit per selector for each virtual orbital and each k.
// An entry finds its connected selectors with a few AND / OR per 32 selectors
// and visits those alone.  Testing every selector against every entry
// instead bound the kernel by integer issue: over 8 generators, 2,000
// selectors and 10.1M entries (14a+14b in 80 MOs) it ran 18.4 ms.  It takes
// 3.8 ms with these masks, the work split evenly over the CTAs, three of them
// resident on an SM and the FP64 instructions of the energies that depend on
// one particle only shared by an item's entries; what is left is the latency
// of the elements' integrals (1.7 ms), the staging of the selectors and the
// lanes that wait for the entry with the most of them.
//
// Banned determinants.  a is dropped when it is in the wave function
// (device hash set of psi_det) or within a double excitation of an earlier
// generator, so that every external determinant is counted once, by the
// first generator that reaches it.  The earlier generators within a
// quadruple excitation of g are listed once per generator; the CTA keeps
// those that lack at most two of mask's electrons.
//
// Energy.  H_aa = diag_H_mat_elem_fock(g, a) (slater_rules.irp.f:1800-1866)
// from the generator's build_fock_tmp (Fock_diag.irp.f:1-98).  For each state,
// e = (sign(delta) sqrt(delta^2 + (2 mat)^2) - delta) / 2 with
// delta = E0 - H_aa.  pt2 sums e.  The buffer gets a with min(0, min_st e)
// when some numerator is non-zero, and keeps the most negative values: a
// device radix sort by value, with ties put in determinant-bit order on the
// host.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <vector>

#include "qpgpu_internal.cuh"

namespace {

constexpr int SBLK = 256;
constexpr int SEL_TILE = 16384;    // FP64 numerators per CTA at most (128 KB of shared memory)
constexpr int SEL_DTILE = 256;     // selectors staged per pass (one word of 32 per warp of the CTA)
constexpr int SEL_DWORDS = SEL_DTILE / 32;
static_assert(SEL_DWORDS == SBLK / 32 && SBLK <= SEL_DTILE, "each warp transposes one word of staged selectors");
constexpr int SEL_MAXST = 8;       // states
constexpr int SEL_SUM = SBLK / 2;  // entries whose energies are summed together, and that units are cut in
constexpr int SEL_MQ = 128;        // single-excitation elements a warp evaluates ahead
constexpr int SEL_MG = 4;          // entries per lane they are collected from
static_assert(SEL_DTILE <= 256 && SEL_MG <= 8, "codes of 3 + 5 + 8 bits");
constexpr int SEL_MAXFG = 2048;    // earlier generators kept per item in shared memory (else read from the global list)

enum { IT_SINGLE = 0, IT_SAME = 1, IT_AB = 2 };

struct SelItem {
  int g;         // generator (psi_det index)
  int gl;        // its position in the generator list of the call
  int kind;      // IT_*
  int spin;      // single / same-spin double: 0 alpha, 1 beta
  int h1, h2;    // holes (1-based); alpha-beta: h1 alpha, h2 beta
  int e0, e1;    // entry range
  int part;      // first of its sums in pt2_part (generators in order)
};

struct SelArgs {
  DevTables t;
  const u64* dets;       // (nint, 2, N)
  const double* coef;    // (N, n_st) row-major (state fastest)
  const double* e0;      // (n_st)
  int n_st;
  int64_t N;
  const SelItem* items;
  const int64_t* ilist_off;  // per listed generator: selectors within a quadruple excitation
  const int* ilist;
  const int64_t* flist_off;  // per listed generator: earlier generators within a quadruple excitation
  const int* flist;
  const double* fock;        // per listed generator: build_fock_tmp, [gl][2][n_mo + 2]
  const int* hslot;          // hash set of psi_det: det index or -1
  uint64_t hmask;
  double* pt2_part;          // [part][n_st]: sums over SEL_SUM entries each
  unsigned long long* n_ext;
  unsigned long long* n_cand;
  uint64_t cap;
  double* cand_val;
  uint64_t* cand_at;         // its unit (high 32 bits) and entry
};

template <int NINT>
__device__ __forceinline__ uint64_t det_hash(const u64* d) {
  uint64_t h = 0x9e3779b97f4a7c15ull;
#pragma unroll
  for (int w = 0; w < 2 * NINT; ++w) {
    h ^= d[w] + 0x9e3779b97f4a7c15ull + (h << 6) + (h >> 2);
    h *= 0xbf58476d1ce4e5b9ull;
  }
  return h ^ (h >> 31);
}

template <int NINT>
__device__ __forceinline__ bool same_det(const u64* a, const u64* b) {
  bool eq = true;
#pragma unroll
  for (int w = 0; w < 2 * NINT; ++w) eq &= a[w] == b[w];
  return eq;
}

template <int NINT>
__global__ void k_hash_insert(const u64* dets, int64_t N, int* slot, uint64_t hmask) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
    const u64* d = dets + i * 2 * NINT;
    uint64_t s = det_hash<NINT>(d) & hmask;
    for (uint64_t probe = 0; probe <= hmask; ++probe) {
      const int prev = atomicCAS(&slot[s], -1, (int)i);
      if (prev == -1) break;
      s = (s + 1) & hmask;
    }
  }
}

template <int NINT>
__device__ __forceinline__ bool in_wf(const SelArgs& A, const u64* a) {
  uint64_t s = det_hash<NINT>(a) & A.hmask;
  for (uint64_t probe = 0; probe <= A.hmask; ++probe) {
    const int i = __ldg(&A.hslot[s]);
    if (i < 0) return false;
    if (same_det<NINT>(A.dets + (int64_t)i * 2 * NINT, a)) return true;
    s = (s + 1) & A.hmask;
  }
  return false;
}

template <int NINT>
__device__ __forceinline__ int exc_deg(const u64* a, const u64* b) {
  int d = 0;
#pragma unroll
  for (int w = 0; w < 2 * NINT; ++w) d += popc64(a[w] ^ b[w]);
  return d >> 1;
}

// per listed generator g = gens[l]: the candidates c < limit (selectors:
// limit = n_sel; earlier generators: limit = g) within a quadruple excitation
// of g, in increasing order.  mode 0 counts into cnt[l], mode 1 fills at off[l].
template <int NINT>
__global__ void __launch_bounds__(SBLK) k_sel_lists(const u64* dets, const int* gens, int n_list, int n_sel,
                                                    int earlier, int mode, int64_t* cnt, const int64_t* off,
                                                    int* out) {
  __shared__ int wsum[SBLK / 32];
  __shared__ int base_s;
  const int l = blockIdx.x;
  if (l >= n_list) return;
  const int g = gens[l];
  u64 gd[2 * NINT];
#pragma unroll
  for (int w = 0; w < 2 * NINT; ++w) gd[w] = dets[(int64_t)g * 2 * NINT + w];
  const int limit = earlier ? g : n_sel;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) base_s = 0;
  __syncthreads();
  for (int c0 = 0; c0 < limit; c0 += SBLK) {
    const int c = c0 + threadIdx.x;
    bool keep = false;
    if (c < limit) keep = exc_deg<NINT>(gd, dets + (int64_t)c * 2 * NINT) <= 4;
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) wsum[warp] = __popc(bal);
    __syncthreads();
    int before = base_s;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    if (mode == 1 && keep) out[off[l] + before + __popc(bal & ((1u << lane) - 1))] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
      int tot = 0;
      for (int w = 0; w < SBLK / 32; ++w) tot += wsum[w];
      base_s += tot;
    }
    __syncthreads();
  }
  if (mode == 0 && threadIdx.x == 0) cnt[l] = base_s;
}

__device__ __forceinline__ bool has_orb(const u64* d, int nint, int spin, int orb) {
  return (d[spin * nint + ((orb - 1) >> 6)] >> ((orb - 1) & 63)) & 1ull;
}

// build_fock_tmp (Fock_diag.irp.f:1-98) of every listed generator:
// f[l][s][i], i = 1..n_mo, and f[l][s][n_mo + 1] = <g|H|g>
// One CTA per generator, a thread per (spin, orbital): each f keeps the order of
// its sum (one thread per generator walked all of them: 443 us for 8
// generators of 28 electrons in 80 orbitals, 12 us now).
template <int NINT>
__global__ void __launch_bounds__(SBLK) k_sel_fock(DevTables t, const u64* dets, const int* gens, int n_list,
                                                   double* fock) {
  __shared__ int occ[2][QPGPU_MAX_MO];
  __shared__ int no[2];
  __shared__ double part[2 * QPGPU_MAX_MO];  // shares of <g|H|g>
  const int l = blockIdx.x;
  if (l >= n_list) return;
  const int n = t.n, st = n + 2;
  const u64* d = dets + (int64_t)gens[l] * 2 * NINT;
  double* f = fock + (int64_t)l * 2 * st;
  if (threadIdx.x < 2) {
    const int s = threadIdx.x;
    int c = 0;
    for (int w = 0; w < NINT; ++w)
      for (u64 x = d[s * NINT + w]; x; x &= x - 1) occ[s][c++] = ctz64(x) + 1 + 64 * w;
    no[s] = c;
  }
  __syncthreads();
  for (int x = threadIdx.x; x < 2 * n; x += SBLK) {
    const int s = x / n, o = 1 - s, i = x % n + 1;
    double v = 0.0, e = 0.0;
    if (has_orb(d, NINT, s, i)) {
      v = tab2(t.h, n, i, i);
      e = tab2(t.h, n, i, i);
      for (int jj = 0; jj < no[s]; ++jj) {
        const int j = occ[s][jj];
        if (i == j) continue;
        v += tab2(t.ja, n, i, j);
        e += 0.5 * tab2(t.ja, n, i, j);
      }
      for (int jj = 0; jj < no[o]; ++jj) {
        const int j = occ[o][jj];
        v += tab2(t.jj, n, i, j);
        if (s == 0) e += tab2(t.jj, n, i, j);
      }
    }
    if (v == 0.0) {  // empty orbitals (the reference tests the sum, not the occupation)
      v += tab2(t.h, n, i, i);
      for (int jj = 0; jj < no[s]; ++jj) v += tab2(t.ja, n, i, occ[s][jj]);
      for (int jj = 0; jj < no[o]; ++jj) v += tab2(t.jj, n, i, occ[o][jj]);
    }
    f[s * st + i] = v;
    part[x] = e;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double e0 = 0.0;
    for (int x = 0; x < 2 * n; ++x) e0 += part[x];
    f[0] = f[st] = 0.0;
    f[n + 1] = e0;
    f[st + n + 1] = e0;
  }
}

// <a|H|D>, generic path (degree from the words; a is the first determinant, E = det_parity of a)
template <int NINT>
__device__ __forceinline__ double ihj(const DevTables& t, const u64* a, const u64* D, const u64* E) {
  int da = 0, db = 0;
#pragma unroll
  for (int w = 0; w < NINT; ++w) {
    da += popc64(a[w] ^ D[w]);
    db += popc64(a[NINT + w] ^ D[NINT + w]);
  }
  if (da + db == 4) {
    if (da == 4) return h_double_spin<NINT>(t, a, D, E, nullptr, nullptr);
    if (db == 4) return h_double_spin<NINT>(t, a + NINT, D + NINT, E + NINT, nullptr, nullptr);
    double s2;
    return h_double_ab<NINT>(t, a, D, E, &s2, nullptr, nullptr);
  }
  if (da + db == 2) return h_mono_spin<NINT>(t, a, D, E, da == 2 ? 1 : 2, nullptr, nullptr);
  if (da + db == 0) return diag_h<NINT>(t, a);
  return 0.0;
}

// every word is written, so the determinant stays in registers
template <int NINT>
__device__ __forceinline__ void set_orb(u64* d, int spin, int orb, bool on) {
  const u64 b = 1ull << ((orb - 1) & 63);
  const int at = spin * NINT + ((orb - 1) >> 6);
#pragma unroll
  for (int w = 0; w < 2 * NINT; ++w)
    if (w == at) d[w] = on ? (d[w] | b) : (d[w] & ~b);
}

// triangular entry e -> (i1 < i2)
__device__ __forceinline__ void tri_decode(int e, int& i1, int& i2) {
  int j = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)e)) * 0.5f);
  while (j * (j - 1) / 2 > e) --j;
  while ((j + 1) * j / 2 <= e) ++j;
  i2 = j;
  i1 = e - j * (j - 1) / 2;
}

// bit c of lane r -> bit r of lane c
__device__ __forceinline__ unsigned transpose32(unsigned x, int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned lo = o == 16 ? 0x0000ffffu : o == 8 ? 0x00ff00ffu : o == 4 ? 0x0f0f0f0fu : o == 2 ? 0x33333333u
                                                                                                   : 0x55555555u;
    const unsigned y = __shfl_xor_sync(0xffffffffu, x, o);
    x = lane & o ? (x & ~lo) | ((y >> o) & lo) : (x & lo) | ((y & lo) << o);
  }
  return x;
}

// the generator without the item's holes
template <int NINT>
__device__ __forceinline__ void item_mask(const SelItem& it, const u64* gd, u64* mask) {
#pragma unroll
  for (int w = 0; w < 2 * NINT; ++w) mask[w] = gd[w];
  if (it.kind == IT_SINGLE) {
    set_orb<NINT>(mask, it.spin, it.h1, false);
  } else if (it.kind == IT_SAME) {
    set_orb<NINT>(mask, it.spin, it.h1, false);
    set_orb<NINT>(mask, it.spin, it.h2, false);
  } else {
    set_orb<NINT>(mask, 0, it.h1, false);
    set_orb<NINT>(mask, 1, it.h2, false);
  }
}

// Work of an item, in matrix elements: with k electrons of the mask missing, a
// selector is connected to every entry (k = 0; singles also k = 1), to those
// that hold one of its three electrons outside the mask (k = 1) or to a few
// (k = 2).  An entry's energy counts as ENTRY_COST elements.  One warp per
// item.
constexpr double ENTRY_COST = 2.5, LIST_COST = 1.5;
template <int NINT>
__global__ void __launch_bounds__(SBLK) k_sel_weigh(SelArgs A, int64_t n_items, float* weight) {
  const int lane = threadIdx.x & 31;
  for (int64_t i = (blockIdx.x * (int64_t)SBLK + threadIdx.x) >> 5; i < n_items; i += ((int64_t)gridDim.x * SBLK) >> 5) {
    const SelItem it = A.items[i];
    u64 mask[2 * NINT];
    item_mask<NINT>(it, A.dets + (int64_t)it.g * 2 * NINT, mask);
    int n0 = 0, n1 = 0, n2 = 0;
    const int64_t i1 = A.ilist_off[it.gl + 1];
    for (int64_t q = A.ilist_off[it.gl] + lane; q < i1; q += 32) {
      const u64* D = A.dets + (int64_t)A.ilist[q] * 2 * NINT;
      int k = 0;
#pragma unroll
      for (int w = 0; w < 2 * NINT; ++w) k += popc64(mask[w] & ~__ldg(&D[w]));
      n0 += k == 0;
      n1 += k == 1;
      n2 += k == 2;
    }
    n0 = __reduce_add_sync(0xffffffffu, n0);
    n1 = __reduce_add_sync(0xffffffffu, n1);
    n2 = __reduce_add_sync(0xffffffffu, n2);
    if (lane == 0) {
      const float ne = (float)(it.e1 - it.e0);
      const float near = it.kind == IT_SINGLE ? ne : fminf(ne, 3.0f * (float)A.t.n);
      weight[i] = ne * ((float)n0 + (float)ENTRY_COST) + (float)n1 * near + 4.0f * (float)n2;
    }
  }
}

template <int NINT>
__global__ void __launch_bounds__(SBLK, 3) k_sel_items(SelArgs A) {
  extern __shared__ double tile[];  // [entry - e0][n_st]
  __shared__ u64 sdet[SEL_DTILE][2 * NINT];
  __shared__ int sidx[SEL_DTILE];
  __shared__ unsigned char sk[SEL_DTILE];
  __shared__ unsigned shas[SEL_DWORDS][2][QPGPU_MAX_MO];  // staged selectors that hold an orbital
  __shared__ unsigned skm[SEL_DWORDS][3];                 // staged selectors with k = 0, 1, 2
  __shared__ int vir[2][QPGPU_MAX_MO];
  __shared__ int nvir[2];
  __shared__ int fgen[SEL_MAXFG];
  __shared__ int nfg;
  __shared__ int wsum[SBLK / 32];
  __shared__ double mono_h[SBLK / 32][SEL_MQ];
  __shared__ unsigned short mono_c[SBLK / 32][SEL_MQ];
  const SelItem it = A.items[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nst = A.n_st, n = A.t.n;
  const u64* gd = A.dets + (int64_t)it.g * 2 * NINT;
  u64 mask[2 * NINT];
  item_mask<NINT>(it, gd, mask);
  if (tid < 2) {
    int c = 0;
    for (int o = 1; o <= n; ++o)
      if (!has_orb(gd, NINT, tid, o)) vir[tid][c++] = o;
    nvir[tid] = c;
  }
  if (tid == 0) nfg = 0;
  __syncthreads();
  // the earlier generators that can reach a determinant of this item
  {
    const int64_t f0 = A.flist_off[it.gl], f1 = A.flist_off[it.gl + 1];
    for (int64_t f = f0 + tid; f < f1; f += SBLK) {
      const int gp = A.flist[f];
      const u64* q = A.dets + (int64_t)gp * 2 * NINT;
      int k = 0;
#pragma unroll
      for (int w = 0; w < 2 * NINT; ++w) k += popc64(mask[w] & ~q[w]);
      if (k <= 2) {
        const int slot = atomicAdd(&nfg, 1);
        if (slot < SEL_MAXFG) fgen[slot] = gp;  // past SEL_MAXFG the bans read the global list
      }
    }
  }
  // owned entries: e = it.e0 + tid + j SBLK
  const int ne = it.e1 - it.e0;
  for (int x = tid; x < ne * nst; x += SBLK) tile[x] = 0.0;
  __syncthreads();
  const int sp1 = it.kind == IT_AB ? 0 : it.spin;  // spin of particle 1
  const int sp2 = it.kind == IT_AB ? 1 : it.spin;  // spin of particle 2
  const bool two = it.kind != IT_SINGLE;
  // an entry's particles: their positions in vir[sp1], vir[sp2] and the orbitals
  auto entry = [&](int e, int& v1, int& v2) {
    if (it.kind == IT_SINGLE) {
      v1 = e;
      v2 = 0;
    } else if (it.kind == IT_SAME) {
      tri_decode(e, v1, v2);
    } else {
      const int nb = nvir[1];
      v1 = e / nb;
      v2 = e - v1 * nb;
    }
  };
  auto particles = [&](int e, int& p1, int& p2) {
    int v1, v2;
    entry(e, v1, v2);
    p1 = vir[sp1][v1];
    p2 = two ? vir[sp2][v2] : 0;
  };
  const int64_t i0 = A.ilist_off[it.gl], i1 = A.ilist_off[it.gl + 1];
  int64_t base = i0;
  while (base < i1) {
    // stage the next selectors with k = |mask \ D| <= 2, in order: blocks of
    // SBLK candidates as long as what they keep fits the tile
    int ns = 0;
    while (base < i1) {
      const int64_t q = base + tid;
      int D = -1, k = 3;
      u64 dd[2 * NINT];
      if (q < i1) {
        D = A.ilist[q];
        k = 0;
#pragma unroll
        for (int w = 0; w < 2 * NINT; ++w) {
          dd[w] = A.dets[(int64_t)D * 2 * NINT + w];
          k += popc64(mask[w] & ~dd[w]);
        }
      }
      const bool keep = k <= 2;
      const unsigned bal = __ballot_sync(0xffffffffu, keep);
      if (lane == 0) wsum[warp] = __popc(bal);
      __syncthreads();
      int before = 0, total = 0;
#pragma unroll
      for (int w = 0; w < SBLK / 32; ++w) {
        before += w < warp ? wsum[w] : 0;
        total += wsum[w];
      }
      __syncthreads();
      if (ns + total > SEL_DTILE) break;  // this block opens the next tile
      if (keep) {
        const int pos = ns + before + __popc(bal & ((1u << lane) - 1));
#pragma unroll
        for (int w = 0; w < 2 * NINT; ++w) sdet[pos][w] = dd[w];
        sidx[pos] = D;
        sk[pos] = (unsigned char)k;
      }
      ns += total;
      base += SBLK;
    }
    __syncthreads();
    const int nw = (ns + 31) >> 5;
    // transposed tile: warp w turns selectors 32 w .. 32 w + 31 into one word
    // per orbital and one per k
    if (warp < nw) {
      const int j = warp * 32 + lane;
      const bool live = j < ns;
#pragma unroll
      for (int c = 0; c < 2 * 2 * NINT; ++c) {  // 32 orbitals each
        const int sp = c / (2 * NINT), part = c % (2 * NINT);
        if (part * 32 >= n) continue;
        const u64 x = live ? sdet[j][sp * NINT + part / 2] : 0ull;
        shas[warp][sp][part * 32 + lane] = transpose32((unsigned)(part & 1 ? x >> 32 : x), lane);
      }
      const int k = live ? sk[j] : 3;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const unsigned bal = __ballot_sync(0xffffffffu, k == q);
        if (lane == 0) skm[warp][q] = bal;
      }
    }
    __syncthreads();
    // every thread: its entries against their connected selectors, in order.
    // deg = k + [p1 not in D] + [p2 not in D] is 1 or 2 for 32 selectors at a
    // time (deg 0: a = D, in the wave function).  The few single excitations
    // (deg 1) are sums over all electrons, whose dozens of FP64 instructions
    // cost a warp the same for one lane as for 32: the warp collects those of
    // its next SEL_MG x 32 entries first and evaluates them side by side.
    auto words = [&](int w, int p1, int p2, unsigned& deg1, unsigned& deg12) {
      const unsigned h1 = shas[w][sp1][p1 - 1], h2 = two ? shas[w][sp2][p2 - 1] : 0xffffffffu;
      const unsigned k0 = skm[w][0], k1 = skm[w][1];
      deg1 = (k0 & (h1 ^ h2)) | (k1 & h1 & h2);
      deg12 = (k0 & ~(h1 & h2)) | (k1 & (h1 | h2)) | (skm[w][2] & h1 & h2);
    };
    auto external = [&](int p1, int p2, u64* a, u64* E) {
#pragma unroll
      for (int w = 0; w < 2 * NINT; ++w) a[w] = mask[w];
      set_orb<NINT>(a, sp1, p1, true);
      if (two) set_orb<NINT>(a, sp2, p2, true);
      det_parity<NINT>(a, E);
    };
    for (int eb = warp * 32; eb < ne; eb += SEL_MG * SBLK) {
      int n1 = 0;
      for (int q = 0; q < SEL_MG; ++q) {
        const int e = eb + q * SBLK + lane;
        if (e >= ne) break;
        int p1, p2;
        particles(it.e0 + e, p1, p2);
        for (int w = 0; w < nw; ++w) {
          unsigned deg1, deg12;
          words(w, p1, p2, deg1, deg12);
          n1 += __popc(deg1);
        }
      }
      int upto = n1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += x;
      }
      const int n1_warp = min(__shfl_sync(0xffffffffu, upto, 31), SEL_MQ);
      int at = upto - n1;
      if (n1_warp > 0) {
        int put = at;
        for (int q = 0; n1 > 0 && q < SEL_MG; ++q) {
          const int e = eb + q * SBLK + lane;
          if (e >= ne) break;
          int p1, p2;
          particles(it.e0 + e, p1, p2);
          for (int w = 0; w < nw; ++w) {
            unsigned deg1, deg12;
            words(w, p1, p2, deg1, deg12);
            for (; deg1; deg1 &= deg1 - 1, ++put)
              if (put < SEL_MQ)
                mono_c[warp][put] = (unsigned short)((q << 13) | (lane << 8) | (w * 32 + __ffs(deg1) - 1));
          }
        }
        __syncwarp();
        for (int i = lane; i < n1_warp; i += 32) {
          const int code = mono_c[warp][i];
          int p1, p2;
          particles(it.e0 + eb + (code >> 13) * SBLK + ((code >> 8) & 31), p1, p2);
          u64 a[2 * NINT], E[2 * NINT], Dw[2 * NINT];
          external(p1, p2, a, E);
#pragma unroll
          for (int x = 0; x < 2 * NINT; ++x) Dw[x] = sdet[code & 255][x];
          bool beta = true;
#pragma unroll
          for (int x = 0; x < NINT; ++x) beta = beta && a[x] == Dw[x];
          mono_h[warp][i] = h_mono_spin<NINT>(A.t, a, Dw, E, beta ? 2 : 1, nullptr, nullptr);
        }
        __syncwarp();
      }
      for (int q = 0; q < SEL_MG; ++q) {
        const int e = eb + q * SBLK + lane;
        if (e >= ne) break;
        int p1, p2;
        particles(it.e0 + e, p1, p2);
        u64 a[2 * NINT], E[2 * NINT];
        external(p1, p2, a, E);
        double* m = tile + (size_t)e * nst;
        double m0 = m[0];
        int w = -1;
        unsigned bits = 0, deg1 = 0;
        while (true) {
          while (bits == 0 && ++w < nw) words(w, p1, p2, deg1, bits);
          if (bits == 0) break;
          const unsigned b = bits & (0u - bits);
          const int j = w * 32 + __ffs(bits) - 1;
          bits ^= b;
          const bool single = deg1 & b;
          at += single;
          double h;
          if (single && at <= SEL_MQ) {
            h = mono_h[warp][at - 1];
          } else {
            u64 Dw[2 * NINT];
#pragma unroll
            for (int x = 0; x < 2 * NINT; ++x) Dw[x] = sdet[j][x];
            h = ihj<NINT>(A.t, a, Dw, E);
          }
          const double* cD = A.coef + (int64_t)sidx[j] * nst;
          m0 = fma(__ldg(&cD[0]), h, m0);
          for (int s = 1; s < nst; ++s) m[s] = fma(__ldg(&cD[s]), h, m[s]);
        }
        m[0] = m0;
      }
      __syncwarp();
    }
    __syncthreads();
  }
  // diag_H_mat_elem_fock (slater_rules.irp.f:1800-1866), holes and particles
  // ascending within a spin as decode_exc lists them: what depends on one
  // particle only is summed once per item, in the same order
  const int st = n + 2;
  const double* F = A.fock + (int64_t)it.gl * 2 * st;
  const double eg = F[n + 1];
  double* const hp1 = mono_h[0];
  double* const hp2 = mono_h[1];
  double* const hq2 = mono_h[2];
  static_assert(SEL_MQ >= QPGPU_MAX_MO, "the particles' shares take the place of the queue");
  const double* pp = it.kind == IT_AB ? A.t.jj : A.t.ja;  // between the two spins of the item
  {
    const double* F1 = F + sp1 * st;
    const double* F2 = F + sp2 * st;
    const int h1 = it.h1, h2 = it.h2;  // same spin: h1 < h2, p1 < p2
    for (int v = tid; v < nvir[sp1]; v += SBLK) {
      const int p1 = vir[sp1][v];
      double x = eg - F1[h1] + (F1[p1] - tab2(A.t.ja, n, h1, p1));
      if (two) x = x - (F2[h2] - tab2(pp, n, h1, h2) + tab2(pp, n, p1, h2));
      hp1[v] = x;
    }
    if (two)
      for (int v = tid; v < nvir[sp2]; v += SBLK) {
        const int p2 = vir[sp2][v];
        hp2[v] = F2[p2] - tab2(pp, n, h1, p2);
        hq2[v] = tab2(A.t.ja, n, h2, p2);
      }
    __syncthreads();
  }
  // energies of this thread's entries, in place of their numerators (zero for
  // an entry that does not count)
  unsigned long long next = 0;
  for (int e = tid; e < ne; e += SBLK) {
    double* m = tile + (size_t)e * nst;
    unsigned long long any = 0;
    for (int s = 0; s < nst; ++s) any |= (unsigned long long)__double_as_longlong(m[s]) << 1;
    if (any == 0) continue;
    int v1, v2;
    entry(it.e0 + e, v1, v2);
    const int p1 = vir[sp1][v1], p2 = two ? vir[sp2][v2] : 0;
    u64 a[2 * NINT];
#pragma unroll
    for (int w = 0; w < 2 * NINT; ++w) a[w] = mask[w];
    set_orb<NINT>(a, sp1, p1, true);
    if (two) set_orb<NINT>(a, sp2, p2, true);
    bool banned = in_wf<NINT>(A, a);
    if (nfg <= SEL_MAXFG) {
      for (int f = 0; f < nfg && !banned; ++f) banned = exc_deg<NINT>(a, A.dets + (int64_t)fgen[f] * 2 * NINT) <= 2;
    } else {  // more earlier generators reach this item than the shared list holds
      for (int64_t f = A.flist_off[it.gl]; f < A.flist_off[it.gl + 1] && !banned; ++f)
        banned = exc_deg<NINT>(a, A.dets + (int64_t)A.flist[f] * 2 * NINT) <= 2;
    }
    if (banned) {
      for (int s = 0; s < nst; ++s) m[s] = 0.0;
      continue;
    }
    ++next;
    double haa = hp1[v1];
    if (two) haa += (hp2[v2] + tab2(pp, n, p1, p2)) - hq2[v2];
    double mine = 0.0;
    for (int s = 0; s < nst; ++s) {
      const double delta = A.e0[s] - haa;
      const double val = m[s] + m[s];
      double tmp = sqrt(delta * delta + val * val);
      if (delta < 0.0) tmp = -tmp;
      const double ev = 0.5 * (tmp - delta);
      m[s] = ev;
      mine = fmin(ev, mine);
    }
    // one atomic for the lanes that are here together
    const unsigned grp = __activemask();
    unsigned long long slot = 0;
    if (lane == __ffs(grp) - 1) slot = atomicAdd(A.n_cand, (unsigned long long)__popc(grp));
    slot = __shfl_sync(grp, slot, __ffs(grp) - 1) + __popc(grp & ((1u << lane) - 1));
    if (slot < A.cap) {
      A.cand_val[slot] = mine;
      A.cand_at[slot] = (uint64_t)blockIdx.x << 32 | (unsigned)(it.e0 + e);
    }
  }
  if (next) atomicAdd(A.n_ext, next);
  // sums over SEL_SUM entries of the item each, whatever unit they are in: how
  // a call's work is split does not show in the bits
  __syncthreads();
  const int nsum = (ne + SEL_SUM - 1) / SEL_SUM;
  for (int x = warp; x < nsum * nst; x += SBLK / 32) {
    const int b = x / nst, s = x - b * nst;
    double acc = 0.0;
#pragma unroll
    for (int q = 0; q < SEL_SUM / 32; ++q) {
      const int e = b * SEL_SUM + 32 * q + lane;
      if (e < ne) acc += tile[(size_t)e * nst + s];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) A.pt2_part[((int64_t)it.part + b) * nst + s] = acc;
  }
}

// detail[l][s] = sum over the parts of listed generator l: one CTA per
// generator and state, strided sums combined in thread order (one thread
// walking 3,248 of them waited 193 us on its loads)
__global__ void __launch_bounds__(SBLK) k_sel_pt2(const double* part, const int64_t* first, int nst, double* detail) {
  __shared__ double red[SBLK];
  const int l = blockIdx.x, s = blockIdx.y;
  double acc = 0.0;
#pragma unroll 8
  for (int64_t i = first[l] + threadIdx.x; i < first[l + 1]; i += SBLK) acc += part[i * nst + s];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int o = SBLK / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) detail[(int64_t)l * nst + s] = red[0];
}

// ascending order of doubles as unsigned keys
__device__ __forceinline__ unsigned long long sel_key(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | (1ull << 63));
}

// The buffer holds a few of millions of candidates.  Two histograms of 12 key
// bits each find the key prefix up to which at least `want` of them lie, and
// only those are sorted (sorting all 10.1M took 0.85 ms and 320 MB).
constexpr int SEL_BINS = 4096;
struct SelCut {
  unsigned long long want, below, prefix, upto;  // below: candidates before the prefix; upto: with it
};

__global__ void __launch_bounds__(SBLK) k_sel_hist(const double* v, uint64_t n, int level, const SelCut* cut,
                                                   unsigned long long* hist) {
  __shared__ unsigned h[SEL_BINS];
  for (int i = threadIdx.x; i < SEL_BINS; i += SBLK) h[i] = 0;
  __syncthreads();
  const unsigned long long prefix = level ? cut->prefix : 0;
  for (uint64_t i = blockIdx.x * (uint64_t)SBLK + threadIdx.x; i < n; i += (uint64_t)gridDim.x * SBLK) {
    const unsigned long long k = sel_key(v[i]);
    if (level == 0)
      atomicAdd(&h[k >> 52], 1u);
    else if ((k >> 52) == prefix)
      atomicAdd(&h[(k >> 40) & (SEL_BINS - 1)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < SEL_BINS; i += SBLK)
    if (h[i]) atomicAdd(&hist[i], (unsigned long long)h[i]);
}

// one block: the first bin that reaches `want`
__global__ void __launch_bounds__(1024) k_sel_pick(const unsigned long long* hist, int level, SelCut* cut) {
  __shared__ unsigned long long part[1024];
  constexpr int PER = SEL_BINS / 1024;
  const int t = threadIdx.x;
  unsigned long long mine = 0;
  for (int i = 0; i < PER; ++i) mine += hist[t * PER + i];
  part[t] = mine;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const unsigned long long x = t >= o ? part[t - o] : 0;
    __syncthreads();
    part[t] += x;
    __syncthreads();
  }
  const unsigned long long want = cut->want, below = level ? cut->below : 0, prefix = level ? cut->prefix : 0;
  __syncthreads();
  unsigned long long at = below + part[t] - mine;
  if (at >= want || below + part[t] < want) return;  // one thread goes on
  for (int i = 0; i < PER; ++i) {
    const unsigned long long c = hist[t * PER + i];
    if (at + c >= want) {
      cut->below = at;
      cut->prefix = prefix << 12 | (unsigned)(t * PER + i);
      cut->upto = at + c;
      return;
    }
    at += c;
  }
}

// keys and numbers of the candidates up to the cut (of all, without one)
__global__ void k_sel_keys(const double* v, uint64_t n, const SelCut* cut, unsigned long long* key, uint64_t* idx,
                           unsigned long long* count) {
  const unsigned long long last = cut ? cut->prefix : 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const unsigned long long k = sel_key(v[i]);
    uint64_t o = i;
    if (cut) {
      if ((k >> 40) > last) continue;
      o = atomicAdd(count, 1ull);
    }
    key[o] = k;
    idx[o] = i;
  }
}

// the head of the sorted candidates, contiguous, as determinants
template <int NINT>
__global__ void k_sel_gather(const uint64_t* idx, uint64_t take, const double* cval, const uint64_t* cat,
                             const SelItem* units, const u64* gens, int n_mo, double* vals, u64* out) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < take; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t j = idx[i];
    vals[i] = cval[j];
    const SelItem it = units[cat[j] >> 32];
    const int e = (int)(unsigned)cat[j];
    const u64* g = gens + (int64_t)it.g * 2 * NINT;
    u64 d[2 * NINT];
    item_mask<NINT>(it, g, d);
    // virtual orbital number v of the generator
    auto vir = [&](int spin, int v) {
      int o = 1;
      for (;; ++o)
        if (!has_orb(g, NINT, spin, o) && v-- == 0) break;
      return o;
    };
    int v1 = e, v2 = 0;
    if (it.kind == IT_SAME) {
      tri_decode(e, v1, v2);
    } else if (it.kind == IT_AB) {
      int nb = n_mo;
      for (int w = 0; w < NINT; ++w) nb -= popc64(g[NINT + w]);
      v1 = e / nb;
      v2 = e - v1 * nb;
    }
    set_orb<NINT>(d, it.kind == IT_AB ? 0 : it.spin, vir(it.kind == IT_AB ? 0 : it.spin, v1), true);
    if (it.kind != IT_SINGLE) set_orb<NINT>(d, it.kind == IT_AB ? 1 : it.spin, vir(it.kind == IT_AB ? 1 : it.spin, v2), true);
    for (int w = 0; w < 2 * NINT; ++w) out[i * 2 * NINT + w] = d[w];
  }
}

struct Dev {
  qpgpu_ctx* c;
  void* p = nullptr;
  ~Dev() { qp_pool_free(c, p); }
};

}  // namespace

// The selection over the listed generators (psi_det indices, each banned by
// every generator before it, listed or not).  pt2 (n_st) sums all of them, in
// the order of the list; per_gen (n_list x n_st, optional) holds each
// generator's share, summed in an order that is the generator's own.  The
// buffer as qpgpu_select_pt2.  Returns the number of buffer entries written or
// a negative status.
static int run_selection(qpgpu_ctx* c, const double* coef, int n_st, const double* e0, int n_sel,
                         const std::vector<int>& gens, int buf_size, double* pt2, double* per_gen,
                         uint64_t* buf_dets, double* buf_vals, int64_t* n_ext) {
  const int64_t N = c->N;
  const int nint = c->nint, n = c->n_mo;
  const int n_list = (int)gens.size();
  cudaStream_t st = c->stream;
  PoolTrim trim{c};
  // host copies of the listed generators (item list)
  std::vector<u64> gdet((size_t)n_list * 2 * nint);
  for (int l = 0; l < n_list; ++l)
    QP_CUDA(c, cudaMemcpyAsync(&gdet[(size_t)l * 2 * nint], c->d_dets + (int64_t)gens[l] * 2 * nint,
                               2 * nint * sizeof(u64), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaStreamSynchronize(st));
  const int tile_entries = SEL_TILE / n_st;
  std::vector<SelItem> items;
  auto push = [&](SelItem it, int ne) {
    for (int a = 0; a < ne; a += tile_entries) {
      it.e0 = a;
      it.e1 = std::min(ne, a + tile_entries);
      items.push_back(it);
    }
  };
  for (int l = 0; l < n_list; ++l) {
    const int g = gens[l];
    std::vector<int> occ[2];
    for (int s = 0; s < 2; ++s)
      for (int o = 1; o <= n; ++o)
        if ((gdet[(size_t)l * 2 * nint + s * nint + ((o - 1) >> 6)] >> ((o - 1) & 63)) & 1ull) occ[s].push_back(o);
    const int nv[2] = {n - (int)occ[0].size(), n - (int)occ[1].size()};
    for (int s = 0; s < 2; ++s)
      for (int h : occ[s]) push(SelItem{g, l, IT_SINGLE, s, h, 0, 0, 0, 0}, nv[s]);
    for (int s = 0; s < 2; ++s)
      for (size_t x = 0; x < occ[s].size(); ++x)
        for (size_t y = x + 1; y < occ[s].size(); ++y)
          push(SelItem{g, l, IT_SAME, s, occ[s][x], occ[s][y], 0, 0, 0}, nv[s] * (nv[s] - 1) / 2);
    for (int ha : occ[0])
      for (int hb : occ[1]) push(SelItem{g, l, IT_AB, 0, ha, hb, 0, 0, 0}, nv[0] * nv[1]);
  }
  const int64_t n_items = (int64_t)items.size();
  for (int s = 0; s < n_st; ++s) pt2[s] = 0.0;
  if (n_ext) *n_ext = 0;
  if (n_items == 0) {
    if (per_gen)
      for (size_t x = 0; x < (size_t)n_list * n_st; ++x) per_gen[x] = 0.0;
    return 0;
  }
  // device arrays
  Dev d_items{c}, d_gens{c}, d_coef{c}, d_e0{c}, d_icnt{c}, d_ioff{c}, d_ilist{c}, d_fcnt{c}, d_foff{c};
  Dev d_flist{c}, d_fock{c}, d_slot{c}, d_part{c}, d_cnt{c}, d_pt2{c}, d_wgt{c}, d_units{c}, d_first{c};
  uint64_t hcap = 1;
  while (hcap < (uint64_t)(2 * N)) hcap <<= 1;
  QP_CUDA(c, qp_pool_alloc(c, &d_items.p, items.size() * sizeof(SelItem)));
  QP_CUDA(c, cudaMemcpyAsync(d_items.p, items.data(), items.size() * sizeof(SelItem), cudaMemcpyHostToDevice, st));
  QP_CUDA(c, qp_pool_alloc(c, &d_wgt.p, items.size() * sizeof(float)));
  QP_CUDA(c, qp_pool_alloc(c, &d_gens.p, n_list * sizeof(int)));
  QP_CUDA(c, cudaMemcpyAsync(d_gens.p, gens.data(), n_list * sizeof(int), cudaMemcpyHostToDevice, st));
  // coefficients: column-major (N, n_st) on the host -> (N, n_st) row-major
  std::vector<double> crow((size_t)N * n_st);
  for (int s = 0; s < n_st; ++s)
    for (int64_t i = 0; i < N; ++i) crow[(size_t)i * n_st + s] = coef[(size_t)s * N + i];
  QP_CUDA(c, qp_pool_alloc(c, &d_coef.p, crow.size() * sizeof(double)));
  QP_CUDA(c, cudaMemcpyAsync(d_coef.p, crow.data(), crow.size() * sizeof(double), cudaMemcpyHostToDevice, st));
  QP_CUDA(c, qp_pool_alloc(c, &d_e0.p, n_st * sizeof(double)));
  QP_CUDA(c, cudaMemcpyAsync(d_e0.p, e0, n_st * sizeof(double), cudaMemcpyHostToDevice, st));
  QP_CUDA(c, qp_pool_alloc(c, &d_slot.p, hcap * sizeof(int)));
  QP_CUDA(c, cudaMemsetAsync(d_slot.p, 0xff, hcap * sizeof(int), st));
  QP_CUDA(c, qp_pool_alloc(c, &d_fock.p, (size_t)n_list * 2 * (n + 2) * sizeof(double)));
  QP_CUDA(c, qp_pool_alloc(c, &d_icnt.p, (n_list + 1) * sizeof(int64_t)));
  QP_CUDA(c, qp_pool_alloc(c, &d_fcnt.p, (n_list + 1) * sizeof(int64_t)));
  QP_CUDA(c, qp_pool_alloc(c, &d_cnt.p, 2 * sizeof(unsigned long long)));
  QP_CUDA(c, qp_pool_alloc(c, &d_pt2.p, (size_t)n_list * n_st * sizeof(double)));
  const u64* dets = c->d_dets;
  const int* dg = (const int*)d_gens.p;
  const int hb = (int)std::min<int64_t>((N + 255) / 256, (int64_t)c->n_sm * 8);
#define QP_SEL_NINT(NI)                                                                                          \
  k_hash_insert<NI><<<hb, 256, 0, st>>>(dets, N, (int*)d_slot.p, hcap - 1);                                     \
  k_sel_lists<NI><<<n_list, SBLK, 0, st>>>(dets, dg, n_list, n_sel, 0, 0, (int64_t*)d_icnt.p, nullptr, nullptr); \
  k_sel_lists<NI><<<n_list, SBLK, 0, st>>>(dets, dg, n_list, n_sel, 1, 0, (int64_t*)d_fcnt.p, nullptr, nullptr); \
  k_sel_fock<NI><<<n_list, SBLK, 0, st>>>(c->tab, dets, dg, n_list, (double*)d_fock.p);
  if (nint == 1) {
    QP_SEL_NINT(1)
  } else {
    QP_SEL_NINT(2)
  }
#undef QP_SEL_NINT
  QP_CUDA(c, cudaGetLastError());
  // list offsets on the host
  std::vector<int64_t> icnt(n_list), fcnt(n_list), ioff(n_list + 1), foff(n_list + 1);
  QP_CUDA(c, cudaMemcpyAsync(icnt.data(), d_icnt.p, n_list * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaMemcpyAsync(fcnt.data(), d_fcnt.p, n_list * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaStreamSynchronize(st));
  ioff[0] = foff[0] = 0;
  for (int l = 0; l < n_list; ++l) {
    ioff[l + 1] = ioff[l] + icnt[l];
    foff[l + 1] = foff[l] + fcnt[l];
  }
  QP_CUDA(c, qp_pool_alloc(c, &d_ioff.p, (n_list + 1) * sizeof(int64_t)));
  QP_CUDA(c, qp_pool_alloc(c, &d_foff.p, (n_list + 1) * sizeof(int64_t)));
  QP_CUDA(c, cudaMemcpyAsync(d_ioff.p, ioff.data(), (n_list + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, st));
  QP_CUDA(c, cudaMemcpyAsync(d_foff.p, foff.data(), (n_list + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, st));
  QP_CUDA(c, qp_pool_alloc(c, &d_ilist.p, std::max<int64_t>(1, ioff[n_list]) * sizeof(int)));
  QP_CUDA(c, qp_pool_alloc(c, &d_flist.p, std::max<int64_t>(1, foff[n_list]) * sizeof(int)));
  // candidates (only when a buffer is asked for): at most one per entry
  uint64_t ub = 0;
  for (const SelItem& it : items) ub += (uint64_t)(it.e1 - it.e0);
  uint64_t cap = buf_size > 0 ? std::min<uint64_t>(ub, 1ull << 28) : 0;  // <= 4.3 GB of candidates
  Dev d_cval{c}, d_cat{c};
  SelArgs A{};
  A.t = c->tab;
  A.dets = dets;
  A.coef = (const double*)d_coef.p;
  A.e0 = (const double*)d_e0.p;
  A.n_st = n_st;
  A.N = N;
  A.items = (const SelItem*)d_items.p;  // the items are weighed, then split into units
  A.ilist_off = (const int64_t*)d_ioff.p;
  A.ilist = (const int*)d_ilist.p;
  A.flist_off = (const int64_t*)d_foff.p;
  A.flist = (const int*)d_flist.p;
  A.fock = (const double*)d_fock.p;
  A.hslot = (const int*)d_slot.p;
  A.hmask = hcap - 1;
  A.n_ext = (unsigned long long*)d_cnt.p;
  A.n_cand = (unsigned long long*)d_cnt.p + 1;
#define QP_SEL_WEIGH(NI)                                                                                           \
  k_sel_lists<NI><<<n_list, SBLK, 0, st>>>(dets, dg, n_list, n_sel, 0, 1, nullptr, (const int64_t*)d_ioff.p,       \
                                           (int*)d_ilist.p);                                                       \
  k_sel_lists<NI><<<n_list, SBLK, 0, st>>>(dets, dg, n_list, n_sel, 1, 1, nullptr, (const int64_t*)d_foff.p,       \
                                           (int*)d_flist.p);                                                       \
  k_sel_weigh<NI><<<(unsigned)((n_items + 7) / 8), SBLK, 0, st>>>(A, n_items, (float*)d_wgt.p);
  if (nint == 1) {
    QP_SEL_WEIGH(1)
  } else {
    QP_SEL_WEIGH(2)
  }
#undef QP_SEL_WEIGH
  QP_CUDA(c, cudaGetLastError());
  std::vector<float> wgt(items.size());
  QP_CUDA(c, cudaMemcpyAsync(wgt.data(), d_wgt.p, items.size() * sizeof(float), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaStreamSynchronize(st));
  // Units: an item whose work is above the share of a CTA is split by entries
  // (in multiples of SEL_SUM), and the heaviest units start first.  The
  // work differs by up to a hundred times between items: the call of the
  // header's example ran 8.0 ms with one CTA per item in their order, the last
  // percent of them alone in the second half of that, and 6.1 ms this way.  A
  // share is at least several times what the staging of a CTA costs; 3, 4, 6
  // and 12 shares per resident CTA took 4.4, 3.8, 3.9 and 4.3 ms.
  constexpr int SHARES = 4;
  double work = 0.0;
  for (float w : wgt) work += w;
  const double staging = LIST_COST * (double)ioff[n_list] / n_list;
  const double share = std::max(work / ((double)c->n_sm * 3 * SHARES), 4.0 * staging);
  std::vector<SelItem> units;
  std::vector<float> uw;
  std::vector<int64_t> part_first(n_list + 1, 0);
  int64_t n_parts = 0;
  for (size_t i = 0; i < items.size(); ++i) {
    SelItem it = items[i];
    const int ne = it.e1 - it.e0, blocks = (ne + SEL_SUM - 1) / SEL_SUM;
    const int parts = (int)std::min<double>(std::ceil(wgt[i] / share), blocks);
    const int step = parts <= 1 ? ne : (blocks + parts - 1) / parts * SEL_SUM;
    for (int a = 0; a < ne; a += step) {
      it.e0 = items[i].e0 + a;
      it.e1 = std::min(items[i].e1, it.e0 + step);
      it.part = (int)(n_parts + a / SEL_SUM);
      units.push_back(it);
      uw.push_back(wgt[i] * (float)(it.e1 - it.e0) / (float)ne);
    }
    n_parts += blocks;
    part_first[it.gl + 1] = n_parts;
  }
  for (int l = 0; l < n_list; ++l) part_first[l + 1] = std::max(part_first[l + 1], part_first[l]);
  const int64_t n_units = (int64_t)units.size();
  {
    std::vector<int> order(n_units);
    for (int64_t i = 0; i < n_units; ++i) order[i] = (int)i;
    std::sort(order.begin(), order.end(), [&](int x, int y) { return uw[x] != uw[y] ? uw[x] > uw[y] : x < y; });
    std::vector<SelItem> by_weight(n_units);
    for (int64_t i = 0; i < n_units; ++i) by_weight[i] = units[order[i]];
    units.swap(by_weight);
  }
  QP_CUDA(c, qp_pool_alloc(c, &d_units.p, n_units * sizeof(SelItem)));
  QP_CUDA(c, cudaMemcpyAsync(d_units.p, units.data(), n_units * sizeof(SelItem), cudaMemcpyHostToDevice, st));
  QP_CUDA(c, qp_pool_alloc(c, &d_part.p, (size_t)n_parts * n_st * sizeof(double)));
  QP_CUDA(c, qp_pool_alloc(c, &d_first.p, (n_list + 1) * sizeof(int64_t)));
  QP_CUDA(c, cudaMemcpyAsync(d_first.p, part_first.data(), (n_list + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, st));
  A.items = (const SelItem*)d_units.p;
  A.pt2_part = (double*)d_part.p;
  // dynamic shared memory: the largest unit's numerator tile, so that several CTAs fit an SM
  int max_ne = 0;
  for (const SelItem& it : units) max_ne = std::max(max_ne, it.e1 - it.e0);
  const size_t smem = (size_t)max_ne * n_st * sizeof(double);
  unsigned long long hcnt[2] = {0, 0};
  for (int attempt = 0; attempt < 2; ++attempt) {
    qp_pool_free(c, d_cval.p);
    qp_pool_free(c, d_cat.p);
    d_cval.p = d_cat.p = nullptr;
    QP_CUDA(c, qp_pool_alloc(c, &d_cval.p, std::max<uint64_t>(1, cap) * sizeof(double)));
    QP_CUDA(c, qp_pool_alloc(c, &d_cat.p, std::max<uint64_t>(1, cap) * sizeof(uint64_t)));
    A.cap = cap;
    A.cand_val = (double*)d_cval.p;
    A.cand_at = (uint64_t*)d_cat.p;
    QP_CUDA(c, cudaMemsetAsync(d_cnt.p, 0, 2 * sizeof(unsigned long long), st));
    // (the attribute is for the largest size: another thread may set it before this one launches)
#define QP_SEL_RUN(NI)                                                                                             \
  QP_CUDA(c, cudaFuncSetAttribute(k_sel_items<NI>, cudaFuncAttributeMaxDynamicSharedMemorySize,                    \
                                  SEL_TILE * (int)sizeof(double)));                                                \
  k_sel_items<NI><<<(unsigned)n_units, SBLK, smem, st>>>(A);
    if (nint == 1) {
      QP_SEL_RUN(1)
    } else {
      QP_SEL_RUN(2)
    }
#undef QP_SEL_RUN
    QP_CUDA(c, cudaGetLastError());
    QP_CUDA(c, cudaMemcpyAsync(hcnt, d_cnt.p, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
    QP_CUDA(c, cudaStreamSynchronize(st));
    if (buf_size == 0 || hcnt[1] <= cap) break;
    cap = hcnt[1];  // every candidate counted: run once more with room for all of them
  }
  k_sel_pt2<<<dim3(n_list, n_st), SBLK, 0, st>>>((const double*)d_part.p, (const int64_t*)d_first.p, n_st,
                                                 (double*)d_pt2.p);
  std::vector<double> detail((size_t)n_list * n_st);
  QP_CUDA(c, cudaMemcpyAsync(detail.data(), d_pt2.p, detail.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
  QP_CUDA(c, cudaStreamSynchronize(st));
  for (int l = 0; l < n_list; ++l)
    for (int s = 0; s < n_st; ++s) pt2[s] += detail[(size_t)l * n_st + s];
  if (per_gen) std::copy(detail.begin(), detail.end(), per_gen);
  if (n_ext) *n_ext = (int64_t)hcnt[0];
  const uint64_t nc = std::min<uint64_t>(hcnt[1], cap);
  int nout = (int)std::min<uint64_t>(nc, (uint64_t)buf_size);
  if (nout > 0) {
    // sort by value on the device; the head (and any tie group crossing its
    // end) goes to the host, where equal values are put in determinant order
    Dev kin{c}, kout{c}, vin{c}, vout{c}, tmp{c}, d_cut{c}, d_hist{c};
    const unsigned grid = (unsigned)std::min<uint64_t>((nc + 255) / 256, (uint64_t)c->n_sm * 8);
    // few candidates are sorted as they are: the cut costs 5 launches and a wait
    const bool cut = nc >= (1u << 17) && (uint64_t)nout + 64 < nc / 8;
    uint64_t m = nc;  // candidates to sort
    if (cut) {
      SelCut h{(unsigned long long)nout + 64, 0, 0, 0};
      QP_CUDA(c, qp_pool_alloc(c, &d_cut.p, sizeof(SelCut)));
      QP_CUDA(c, qp_pool_alloc(c, &d_hist.p, (2 * SEL_BINS + 1) * sizeof(unsigned long long)));
      QP_CUDA(c, cudaMemcpyAsync(d_cut.p, &h, sizeof(h), cudaMemcpyHostToDevice, st));
      QP_CUDA(c, cudaMemsetAsync(d_hist.p, 0, (2 * SEL_BINS + 1) * sizeof(unsigned long long), st));
      for (int level = 0; level < 2; ++level) {
        unsigned long long* hist = (unsigned long long*)d_hist.p + level * SEL_BINS;
        k_sel_hist<<<grid, SBLK, 0, st>>>((const double*)d_cval.p, nc, level, (const SelCut*)d_cut.p, hist);
        k_sel_pick<<<1, 1024, 0, st>>>(hist, level, (SelCut*)d_cut.p);
      }
      QP_CUDA(c, cudaMemcpyAsync(&h, d_cut.p, sizeof(h), cudaMemcpyDeviceToHost, st));
      QP_CUDA(c, cudaStreamSynchronize(st));
      m = h.upto;
    }
    QP_CUDA(c, qp_pool_alloc(c, &kin.p, m * 8));
    QP_CUDA(c, qp_pool_alloc(c, &kout.p, m * 8));
    QP_CUDA(c, qp_pool_alloc(c, &vin.p, m * 8));
    QP_CUDA(c, qp_pool_alloc(c, &vout.p, m * 8));
    k_sel_keys<<<grid, 256, 0, st>>>((const double*)d_cval.p, nc, cut ? (const SelCut*)d_cut.p : nullptr,
                                     (unsigned long long*)kin.p, (uint64_t*)vin.p,
                                     cut ? (unsigned long long*)d_hist.p + 2 * SEL_BINS : nullptr);
    size_t tb = 0;
    QP_CUDA(c, cub::DeviceRadixSort::SortPairs(nullptr, tb, (unsigned long long*)kin.p, (unsigned long long*)kout.p,
                                               (uint64_t*)vin.p, (uint64_t*)vout.p, (int64_t)m, 0, 64, st));
    QP_CUDA(c, qp_pool_alloc(c, &tmp.p, tb));
    QP_CUDA(c, cub::DeviceRadixSort::SortPairs(tmp.p, tb, (unsigned long long*)kin.p, (unsigned long long*)kout.p,
                                               (uint64_t*)vin.p, (uint64_t*)vout.p, (int64_t)m, 0, 64, st));
    std::vector<unsigned long long> keys;
    uint64_t take = std::min<uint64_t>(m, (uint64_t)nout + 64);
    while (true) {  // grow the head until it ends past the tie group of entry nout - 1
      keys.resize(take);
      QP_CUDA(c, cudaMemcpyAsync(keys.data(), kout.p, take * 8, cudaMemcpyDeviceToHost, st));
      QP_CUDA(c, cudaStreamSynchronize(st));
      if (take == m || keys[take - 1] != keys[nout - 1]) break;
      take = std::min<uint64_t>(m, take * 2);
    }
    std::vector<double> vals(take);
    std::vector<u64> dts(take * 2 * nint);
    Dev gv{c}, gd{c};
    QP_CUDA(c, qp_pool_alloc(c, &gv.p, take * sizeof(double)));
    QP_CUDA(c, qp_pool_alloc(c, &gd.p, take * 2 * nint * sizeof(u64)));
    const unsigned ggrid = (unsigned)std::min<uint64_t>((take + 127) / 128, (uint64_t)c->n_sm * 8);
#define QP_SEL_GATHER(NI)                                                                                           \
  k_sel_gather<NI><<<ggrid, 128, 0, st>>>((const uint64_t*)vout.p, take, (const double*)d_cval.p,                   \
                                          (const uint64_t*)d_cat.p, (const SelItem*)d_units.p, dets, n,             \
                                          (double*)gv.p, (u64*)gd.p);
    if (nint == 1) {
      QP_SEL_GATHER(1)
    } else {
      QP_SEL_GATHER(2)
    }
#undef QP_SEL_GATHER
    QP_CUDA(c, cudaGetLastError());
    QP_CUDA(c, cudaMemcpyAsync(vals.data(), gv.p, take * sizeof(double), cudaMemcpyDeviceToHost, st));
    QP_CUDA(c, cudaMemcpyAsync(dts.data(), gd.p, take * 2 * nint * sizeof(u64), cudaMemcpyDeviceToHost, st));
    QP_CUDA(c, cudaStreamSynchronize(st));
    std::vector<uint64_t> ord(take);
    for (uint64_t i = 0; i < take; ++i) ord[i] = i;
    std::stable_sort(ord.begin(), ord.end(), [&](uint64_t x, uint64_t y) {
      if (vals[x] != vals[y]) return vals[x] < vals[y];
      for (int w = 0; w < 2 * nint; ++w)
        if (dts[x * 2 * nint + w] != dts[y * 2 * nint + w]) return dts[x * 2 * nint + w] < dts[y * 2 * nint + w];
      return false;
    });
    for (int i = 0; i < nout; ++i) {
      buf_vals[i] = vals[ord[i]];
      for (int w = 0; w < 2 * nint; ++w) buf_dets[(size_t)i * 2 * nint + w] = dts[ord[i] * 2 * nint + w];
    }
  }
  QP_CUDA(c, cudaStreamSynchronize(st));
  return nout;
}

extern "C" int qpgpu_select_pt2(qpgpu_ctx* c, const double* coef, int n_st, const double* e0, int n_gen, int n_sel,
                                int buf_size, double* pt2, uint64_t* buf_dets, double* buf_vals, int64_t* n_ext) {
  if (!c) return QPGPU_ERR_ARG;
  if (!coef || !e0 || !pt2 || n_st < 1 || n_st > SEL_MAXST || buf_size < 0 ||
      (buf_size > 0 && (!buf_dets || !buf_vals)))
    return qpgpu_fail(c, QPGPU_ERR_ARG, "select_pt2: bad arguments (1 <= n_st <= 8, buffers for buf_size > 0)");
  std::lock_guard<std::mutex> lk(c->mu);
  if (!c->have_ints || !c->have_dets)
    return qpgpu_fail(c, QPGPU_ERR_STATE, "select_pt2: integrals and determinants first");
  if (n_gen < 1 || n_gen > n_sel || n_sel > c->N)
    return qpgpu_fail(c, QPGPU_ERR_ARG, "select_pt2: need 1 <= n_gen <= n_sel <= N_det");
  std::vector<int> gens(n_gen);
  for (int g = 0; g < n_gen; ++g) gens[g] = g;
  return run_selection(c, coef, n_st, e0, n_sel, gens, buf_size, pt2, nullptr, buf_dets, buf_vals, n_ext);
}

extern "C" int qpgpu_pt2_generators(qpgpu_ctx* c, const double* coef, int n_st, const double* e0, int n_sel,
                                    const int32_t* gens, int n_list, double* pt2_detail) {
  if (!c) return QPGPU_ERR_ARG;
  if (!coef || !e0 || !gens || !pt2_detail || n_st < 1 || n_st > SEL_MAXST || n_list < 0)
    return qpgpu_fail(c, QPGPU_ERR_ARG, "pt2_generators: bad arguments (1 <= n_st <= 8)");
  std::lock_guard<std::mutex> lk(c->mu);
  if (!c->have_ints || !c->have_dets)
    return qpgpu_fail(c, QPGPU_ERR_STATE, "pt2_generators: integrals and determinants first");
  if (n_sel < 1 || n_sel > c->N) return qpgpu_fail(c, QPGPU_ERR_ARG, "pt2_generators: need 1 <= n_sel <= N_det");
  std::vector<int> g(gens, gens + n_list);
  for (int x : g)
    if (x < 0 || x >= n_sel) return qpgpu_fail(c, QPGPU_ERR_ARG, "pt2_generators: generator outside 0..n_sel-1");
  if (n_list == 0) return QPGPU_OK;
  std::vector<double> tot(n_st);
  const int rc = run_selection(c, coef, n_st, e0, n_sel, g, 0, tot.data(), pt2_detail, nullptr, nullptr, nullptr);
  return rc < 0 ? rc : QPGPU_OK;
}
