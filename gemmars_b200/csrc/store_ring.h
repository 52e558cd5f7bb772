// The turns of the pieces of shared memory through which a warp's results leave (gemm_tc.cu), as plain C++: the kernels and a host
// program run the same code.
#pragma once

#ifdef __CUDACC__
#define GB_RING_FN __device__ __forceinline__
#else
#define GB_RING_FN inline
#endif

// PIECES pieces in turn.  The requests of the thread that sends them (`lead`) form one group a piece, in their order, so that
// "all but the last PIECES - 1 groups have been read" says that the piece to fill next is free.  A piece that holds nothing of
// the result (a tile's features beyond its last one) is a group too, an empty one: were it left out, the wait would leave one
// request more in flight than it is meant to, which may still be reading the piece.
template <int PIECES>
struct StoreRing {
  unsigned posted = 0;
  GB_RING_FN unsigned place() const { return posted % PIECES; }
  // before the piece at place() is filled
  template <typename Queue>
  GB_RING_FN void reuse(bool lead, Queue queue) const {
    if (lead && posted >= PIECES) queue.template wait_read<PIECES - 1>();
  }
  // after it has been filled: `send` makes its requests if there is something of the result in it
  template <typename Queue, typename Send>
  GB_RING_FN void post(bool lead, bool there, Queue queue, Send send) {
    if (lead) {
      if (there) send();
      queue.commit();
    }
    ++posted;
  }
};
