// The walk of k_lincomb_oz's load warp over its ring of block slots, apart
// from the copies and barriers themselves (Io: those of the kernel, or a model
// of them on the host).
//
// A tile t is nb blocks, block b goes to the next of nslots slots (nb ..
// 2 nb), and a slot is free once the K step that read its last block is cut:
//   io.cut(step)        waits for that step of the whole run; false: gave up
//   io.copy(t, b, slot) announces the block's bytes on tile t's barrier (two
//                       barriers, of the even and of the odd tiles) and
//                       starts its copy
//   io.finish(t)        the tile's arrival: from here its phase can complete
//   io.drain(t)         waits until tile t's copies have landed
// Nothing may be on its way when the walk returns, also when it gives up
// inside a tile.  That tile's barrier then counts the bytes of the blocks that
// were started, no others (they are announced one by one), and gets its
// arrival.  When not even the tile's first slot came free the barrier may
// still be in the phase of tile t - 2 and is left alone.
#pragma once

#ifdef __CUDACC__
#define QP_RING_HD __device__ __forceinline__
#else
#define QP_RING_HD inline
#endif

template <class Io>
QP_RING_HD bool block_ring_load(Io& io, int ntile, int nb, int nslots, int nsd, int nks, int ks) {
  int started = 0, slot = 0;  // tiles with copies on their way; next slot
  bool ok = true;
  for (int t = 0; t < ntile && ok; ++t) {
    for (int b = 0; b < nb; ++b) {
      const int old = t * nb + b - nslots;  // the slot's last block
      if (old >= 0) {
        const int ot = old / nb, ob = old - ot * nb;
        ok = io.cut(ot * nks + ((ob + 1) * nsd - 1) / ks);
        if (!ok) break;
      }
      started = t + 1;
      io.copy(t, b, slot);
      if (++slot == nslots) slot = 0;
    }
    if (started == t + 1) io.finish(t);
  }
  for (int t = started > 2 ? started - 2 : 0; t < started; ++t) io.drain(t);
  return ok;
}
