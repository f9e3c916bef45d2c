// The walk of k_lincomb_oz's load warp over its ring of block slots, apart
// from the copies and barriers themselves (Io: those of the kernel, or a model
// of them on the host).
//
// A tile t is nb blocks, block b goes to the next of nslots slots (nb ..
// 2 nb), and a slot is free once the K step that read its last block is cut:
//   io.begin(t)            before the first block of a tile
//   io.cut(step)           waits for that step of the whole run and gives the
//                          number of steps cut (more than `step`), or 0: gave up
//   io.copy(t, b, n, slot) announces the bytes of blocks b .. b + n - 1 on tile
//                          t's barrier (two barriers, of the even and of the
//                          odd tiles) and starts their copies, into the n slots
//                          from `slot` on
//   io.finish(t)           the tile's arrival: from here its phase can complete
//   io.drain(t)            waits until tile t's copies have landed
// The blocks whose slots are free already go together: a K step of KS columns
// frees KS / nsd of them, and narrow blocks started one by one (a wait, an
// announcement and a copy each) took longer than their tile's cut (128 blocks
// of one column).  The warp shares its scheduler with busy ones, so that every
// instruction between a free slot and its copy is felt: the places are counted
// on, with no division by nb or nsd.
// Nothing may be on its way when the walk returns, also when it gives up
// inside a tile.  That tile's barrier then counts the bytes of the blocks that
// were started, no others, and gets its arrival.  When not even the tile's
// first slot came free the barrier may still be in the phase of tile t - 2 and
// is left alone.
#pragma once

#ifdef __CUDACC__
#define QP_RING_HD __device__ __forceinline__
#else
#define QP_RING_HD inline
#endif

template <int KS, class Io>
QP_RING_HD bool block_ring_load(Io& io, int ntile, int nb, int nslots, int nsd, int nks) {
  const int m = nb * nsd;
  const float per_col = 1.0f / (float)nsd;
  int started = 0, slot = 0;  // tiles with copies on their way; next slot
  int fresh = nslots;         // slots not used yet
  // after these: the block that the next slot held last, of the tile whose
  // first K step is step0, by its number and its first column
  int step0 = 0, ob = 0, ocol = 0;
  int done = 0;  // K steps known to be cut
  bool ok = true;
  for (int t = 0; t < ntile && ok; ++t) {
    for (int b = 0; b < nb;) {
      int n = fresh;
      if (fresh == 0) {
        const int step = step0 + (int)((unsigned)(ocol + nsd - 1) / KS);
        if (done <= step) {
          done = io.cut(step);
          ok = done > step;
          if (!ok) break;
        }
        const int cut = (done - step0) * KS;  // columns of that tile that are cut
        n = cut >= m ? nb - ob : (int)(((float)(cut - ocol) + 0.5f) * per_col);
      }
      n = n < nb - b ? n : nb - b;
      n = n < nslots - slot ? n : nslots - slot;
      if (b == 0) io.begin(t);
      started = t + 1;
      io.copy(t, b, n, slot);
      slot = slot + n == nslots ? 0 : slot + n;
      b += n;
      if (fresh > 0) {
        fresh -= n;
      } else {
        ob += n;
        ocol += n * nsd;
        if (ob == nb) {
          ob = ocol = 0;
          step0 += nks;
        }
      }
    }
    if (started == t + 1) io.finish(t);
  }
  for (int t = started > 2 ? started - 2 : 0; t < started; ++t) io.drain(t);
  return ok;
}
