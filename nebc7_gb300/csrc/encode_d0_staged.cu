/* Staged encode kernels: exact differences (kDenoise 0: the precise preset);
   one kernel per pass, everything but the refinement's kinds inlined. */
#define NEBC7_PASS __forceinline__
#define NEBC7_SHARED __forceinline__
#define NEBC7_ONCE __noinline__
#include "bc7_staged_entry.cuh"

NEBC7_INSTANTIATE_STAGED(0)
