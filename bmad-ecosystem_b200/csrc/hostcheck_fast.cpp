// hostcheck_fast.cpp -- TEST-ONLY: the host check build (hostcheck.cpp) with the element forms of
// fastmaps.cuh, the arithmetic of the default device build up to its libm and the last bits of its
// hardware reciprocal approximations (replaced here by single-precision ones, refined the same way).
#define BG_FAST_MAPS 1
#define bmadgpu_hostcheck_track bmadgpu_hostcheck_fast_track
#define bmadgpu_hostcheck_last_error bmadgpu_hostcheck_fast_last_error
#include "hostcheck.cpp"
