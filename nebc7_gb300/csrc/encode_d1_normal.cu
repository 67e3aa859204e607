/* KEncode instantiation: differences halved (kDenoise 1), draft, refinement and
   full-search passes.  Everything but the once-run passes inlined, 255 registers
   and two CTAs per SM: the default preset's time is in one refinement, which
   out of line (four CTAs) spends it on the stack.  The allocation-free entry,
   1024x1024 photo: 8.7 -> 4.4 ms, 512x512 3.4 -> 1.8; alpha 512x512 95 -> 67 ms;
   a 256x256 gradient, mostly draft, 0.25 -> 0.30. */
#define NEBC7_SINGLE_CTAS 2
#define NEBC7_PASS __forceinline__
#define NEBC7_SHARED __forceinline__
#define NEBC7_ONCE __noinline__
#include "bc7_encode_entry.cuh"

NEBC7_INSTANTIATE_ENCODE(1, true)
