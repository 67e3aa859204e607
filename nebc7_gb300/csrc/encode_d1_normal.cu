/* KEncode instantiation: differences halved (kDenoise 1), draft, refinement and
   full-search passes; 255 registers and two CTAs per SM.  The default preset's
   time is in one refinement, which with the registers of four CTAs spends it on
   spills: the allocation-free entry, 512x512 photo 3.41 -> 2.39 ms, 1024x1024 8.80
   -> 5.64; alpha 512x512 95.6 -> 84.5; a 256x256 gradient, mostly draft, 0.24 ->
   0.33.  All inlined, the photos take 1.81 and 4.34 ms, but the thread's stack
   of 5.4 KB makes the first launch reserve 1.4 GB of device memory instead of
   0.26. */
#define NEBC7_SINGLE_CTAS 2
#define NEBC7_PASS __noinline__
#define NEBC7_ONCE __noinline__
#include "bc7_encode_entry.cuh"

NEBC7_INSTANTIATE_ENCODE(1, true)
