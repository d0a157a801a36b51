// The decode kernel of attn_mma.cu for a token whose Q, new rows, positions and slots are read straight out of pinned host
// memory: each CTA fetches its sequence's position, starts its K/V stream and then brings Q into shared memory once for all of
// its warps.  A kernel of its own, because the checks in the other cost launches of 5 us one or two hundredths.
#define VFKV_HOST_INPUTS 1
#include "attn_mma.cu"
