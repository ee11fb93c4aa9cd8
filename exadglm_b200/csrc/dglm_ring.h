// The tiles of a tile buffer ring, in plain C++ (host tests compile it too).
#pragma once

#ifdef __CUDACC__
#define DGLM_HD __host__ __device__ __forceinline__
#else
#define DGLM_HD inline
#endif

namespace dglm {

// A mover warp of a ring of NB buffers serves tiles it = mw, mw + NM, ...
// (NM movers, NM divides NB): at iteration `it` it waits until tile it - NB is
// done with the buffer, and then loads tile `it` there.  When that wait runs
// out, the loads of every tile since it - NB, that one included, may still be
// on their way; settle(q) is called for each of them, oldest first.
template <int NB, int NM, class Settle>
DGLM_HD void mover_in_flight(int it, int total, Settle settle) {
  static_assert(NB % NM == 0, "a mover keeps to its buffers");
  for (int q = it - NB; q < it && q < total; q += NM)
    if (q >= 0) settle(q);
}

}  // namespace dglm
