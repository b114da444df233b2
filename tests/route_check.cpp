// svo_route.h (shocovox_gb300/csrc) for tests/test_routes_host.py, through plain C functions.
#include "../shocovox_gb300/csrc/svo_route.h"

extern "C" {

int route_aligned(const svo_rays* rays, const svo_hits* hits) { return svo::arrays_aligned(*rays, *hits) ? 1 : 0; }

int route_overlap(const svo_rays* rays, const svo_hits* hits, uint64_t n) { return svo::hits_over_rays(*rays, *hits, n) ? 1 : 0; }

}  // extern "C"
