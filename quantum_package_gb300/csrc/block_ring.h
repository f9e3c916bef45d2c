// The walk of k_lincomb_oz's load warp over its ring of block slots, apart
// from the copies and barriers themselves (Io: those of the kernel, or a model
// of them on the host).
//
// A tile t is nb blocks, block b goes to the next of nslots slots (nb ..
// 2 nb), and a slot is free once the K step that read its last block is cut:
//   io.cut(step)           waits for that step of the whole run and gives the
//                          number of steps cut (more than `step`), or 0: gave up
//   io.copy(t, b, n, slot) announces the bytes of blocks b .. b + n - 1 on tile
//                          t's barrier (two barriers, of the even and of the
//                          odd tiles) and starts their copies, into the n slots
//                          from `slot` on
//   io.finish(t)           the tile's arrival: from here its phase can complete
//   io.drain(t)            waits until tile t's copies have landed
// The blocks whose slots are free already go together: a K step frees 16 / nsd
// of them, and narrow blocks started one by one (a wait, an announcement and a
// copy each) took longer than their tile's cut (128 blocks of one column).
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

template <class Io>
QP_RING_HD bool block_ring_load(Io& io, int ntile, int nb, int nslots, int nsd, int nks, int ks) {
  int started = 0, slot = 0;  // tiles with copies on their way; next slot
  int done = 0;               // K steps known to be cut
  bool ok = true;
  for (int t = 0; t < ntile && ok; ++t) {
    for (int b = 0; b < nb;) {
      // the slots' last blocks: old, old + 1, ... of tile ot
      const int old = t * nb + b - nslots;
      int n = nb - b < -old ? nb - b : -old;  // slots not used yet
      if (old >= 0) {
        const int ot = old / nb, ob = old - ot * nb;
        const int step = ot * nks + ((ob + 1) * nsd - 1) / ks;
        if (done <= step) {
          done = io.cut(step);
          ok = done > step;
          if (!ok) break;
        }
        const int cut_cols = (done - ot * nks) * ks;  // columns of tile ot that are cut
        n = (cut_cols < nb * nsd ? cut_cols / nsd : nb) - ob;
        n = n < nb - b ? n : nb - b;
      }
      started = t + 1;
      n = n < nslots - slot ? n : nslots - slot;
      io.copy(t, b, n, slot);
      slot = slot + n == nslots ? 0 : slot + n;
      b += n;
    }
    if (started == t + 1) io.finish(t);
  }
  for (int t = started > 2 ? started - 2 : 0; t < started; ++t) io.drain(t);
  return ok;
}
