// The loading lane's walk over the ring of decoder_rows.cuh: plain C++, so that the host can go through
// every way in which it may end.
#pragma once

#ifdef __CUDACC__
#define SPSATTN_RING_FN __device__ __forceinline__
#else
#define SPSATTN_RING_FN inline
#endif

namespace spsattn {

// Chunks [0, first) are under way in stages 0, 1, ...  Asks for the rest as stages come free; wait_free
// returns false where the step is given up.  Returns how many chunks were asked for.
template <class WaitFree, class Load>
SPSATTN_RING_FN int rows_feed(int first, int chunks, int stages, WaitFree wait_free, Load load) {
  int asked = first;
  for (int st = 0, phase = 0; asked < chunks; ++asked) {
    if (!wait_free(st, phase)) break;
    load(st, asked);
    if (++st == stages) st = 0, phase ^= 1;
  }
  return asked;
}

// The last copy of every stage, when `asked` chunks were asked for: a block that gave up, whoever of it did, leaves
// its shared memory to another only behind these.
template <class WaitLanded>
SPSATTN_RING_FN void rows_landed(int asked, int stages, WaitLanded wait_landed) {
  for (int j = asked > stages ? asked - stages : 0; j < asked; ++j) wait_landed(j % stages, (j / stages) & 1);
}

}  // namespace spsattn
