// Completion counters of the persistent kernels: 32-bit device words that only grow, modulo 2^32.
// Plain C++ besides the annotation, so that the host compiles the kernels' own rule for its tests.
#pragma once

#ifdef __CUDACC__
#define IANE_GB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define IANE_GB_HOST_DEVICE inline
#endif

namespace iane_gb {

// Whether a counter that reads `have` has come as far as `need`. Both may have passed 2^32: what
// counts is the difference, right while the two are less than 2^31 apart.
IANE_GB_HOST_DEVICE bool counter_reached(unsigned int have, unsigned int need)
{
	return static_cast<int>(have - need) >= 0;
}

// Completions of an image's phases before `phase` in a batched run: every tile of a phase counts
// once for each of its four warps. 4 x tiles x phases passes 2^32 within the runs that are accepted
// (2^31 items of up to four tiles); a counter is at most a phase ahead of what is asked of it
// (4 x tiles, which 2^31 bounds for any image that fits in memory) and, as items are taken in order,
// never further behind than the tiles that the CTAs of a launch hold.
IANE_GB_HOST_DEVICE unsigned int batch_need(int phase, int image_tiles)
{
	return static_cast<unsigned int>(phase) * 4u * static_cast<unsigned int>(image_tiles);
}

}  // namespace iane_gb
