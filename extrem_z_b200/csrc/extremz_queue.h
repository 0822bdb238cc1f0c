// Work queue of a search whose blocks find more work as they go (the tile search
// of light manifold rounds, k_touched_tiles): blocks take entries by ticket, push
// what they find, and leave once nothing is left and nobody can find more.  Plain
// C++ over the operations of Q, so that the host can run it on a model of the
// device's memory order.
//
// Q offers: ticket(), place() and finished() (atomic increments of the tickets
// given out, the entries pushed, the entries done; finished() with release order,
// after the block's pushes), done() (acquire order), pushed(), dense(), entry(i),
// store(i, e), ask_dense() (all relaxed) and pause().
#pragma once

#if defined(__CUDACC__)
#define EXTREMZ_HD __host__ __device__ __forceinline__
#else
#define EXTREMZ_HD inline
#endif

namespace extremz {

// The next entry for a block of a queue of `cap` places whose entries carry
// `stamp` in their high half, or -1 when there is none left.  Entry h belongs to
// the block with ticket h, which waits for it only while another block still works
// on one, and at most `limit` times; then it asks for the dense pass, after which
// everyone leaves.
template <class Q>
EXTREMZ_HD int queue_take(Q& q, unsigned stamp, int cap, int limit) {
  const int h = q.ticket();
  for (int spin = 0; spin <= limit; ++spin) {
    if (q.dense()) return -1;
    // (A block sees an entry counted before it takes it, so that what it releases
    // with finished() counts the entry: its stamp alone would not do.)
    if (q.pushed() > h && h < cap) {  // the entry may still be on its way
      const unsigned long long e = q.entry(h);
      if ((unsigned)(e >> 32) == stamp) return (int)(unsigned)e;
    } else {
      // Everything pushed is done: nobody can push more.  `done` comes first, with
      // acquire order, so that `pushed` counts all that the finished blocks pushed.
      // An older `pushed` could equal a newer `done` while entries are open; the
      // block would leave with the ticket of one, and the last block to push would
      // wait for that one up to the limit.
      const int done = q.done();
      if (done == q.pushed()) return -1;
    }
    q.pause();
  }
  q.ask_dense();
  return -1;
}

// Pushes a tile; past `max` places the dense pass takes over.
template <class Q>
EXTREMZ_HD void queue_push(Q& q, unsigned stamp, int tile, int max) {
  const int at = q.place();
  if (at < max) q.store(at, (unsigned long long)stamp << 32 | (unsigned)tile);
  else q.ask_dense();
}

}  // namespace extremz
