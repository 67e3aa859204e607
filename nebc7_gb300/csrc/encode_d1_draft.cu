/* KEncode instantiation: differences halved (kDenoise 1), draft passes only, all
   inlined: with the fast passes and the final pack out of line, photos and alpha
   textures of 64x64 took 331 us instead of 312 and 304 a call, 4096x4096 ones 3.22
   ms instead of 3.18 and 42.4 instead of 40.8. */
#define NEBC7_SHARED
#include "bc7_encode_entry.cuh"

NEBC7_INSTANTIATE_ENCODE(1, false)
