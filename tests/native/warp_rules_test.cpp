// The work-sizing rules of the persistent kernels (warp_rules.h) as C calls.
#include "warp_rules.h"

extern "C" uint32_t wr_lanes_for(uint32_t n, uint32_t warps) { return phc::lanes_for(n, warps); }
extern "C" uint32_t wr_refill_lanes(uint32_t refill, uint32_t per_warp) { return phc::refill_lanes(refill, per_warp); }
extern "C" uint32_t wr_brief_lanes(uint32_t n, uint32_t warps) { return phc::brief_lanes(n, warps); }
