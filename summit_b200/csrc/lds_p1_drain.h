// The end of phase 1's stage ring after an abort (free of CUDA types, so that the
// CPU tests compile it as it is).
#pragma once

#ifdef __CUDACC__
#define LDS_DEV __device__ __forceinline__
#else
#define LDS_DEV inline
#endif

namespace lds {
namespace umma {

// A stage's barrier completes with the weight copy's bytes and one arrival of each
// of the step's decoder warps (set step % sets, set_warps of them).  Decoders that
// give up leave the steps issued since without theirs, and the producer, which may
// not exit before its copies have landed, would wait for each of up to `nst` stages
// until the wait limit.  Once every decoder warp has left its loop, next(w) being the
// first step that warp w did not arrive for, the producer arrives in their place on
// the stages of its last nst steps, whose barriers complete when the bytes are there.
template <class Next, class Arrive>
LDS_DEV void p1_settle(int issued, int nst, int sets, int set_warps, Next next, Arrive arrive) {
    for (int j = issued > nst ? issued - nst : 0; j < issued; ++j)
        for (int u = 0; u < set_warps; ++u)
            if (next((j % sets) * set_warps + u) <= j) arrive(j % nst);
}

}  // namespace umma
}  // namespace lds
