// Bookkeeping of a TMA ring that needs no device: compiles as plain C++ too.
#pragma once

#ifdef __CUDACC__
#define CA_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define CA_HOST_DEVICE inline
#endif

namespace ca {

// Calls wait(stage, parity) for every ring entry whose copies may still be in flight: the last entry ISSUED to each
// stage (an entry that was given up on before its copies were issued is none of them).  An earlier entry of a stage
// has landed, since its consumer released the stage before the next one was issued.
template <typename Wait>
CA_HOST_DEVICE void drain_ring(int issued, int stages, Wait wait) {
  for (int e = issued > stages ? issued - stages : 0; e < issued; ++e) wait(e % stages, static_cast<unsigned>((e / stages) & 1));
}

}  // namespace ca
