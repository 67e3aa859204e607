/* KEncode instantiation: exact differences (kDenoise 0), draft passes only. */
#define NEBC7_SHARED
/* the fast passes and the final pack out of line, each with its own register
   allocation: photos of 4096x4096 without error stepping 182 ms instead of 191,
   of 1024x1024 11.5 instead of 12.1 (alpha textures 199 instead of 193 ms, with
   steps the same) */
#define NEBC7_ONCE __noinline__
#include "bc7_encode_entry.cuh"

NEBC7_INSTANTIATE_ENCODE(0, false)
