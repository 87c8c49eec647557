// How the kernels whose warps march down z split a volume (plain C++: the host tests use it too).
#pragma once

namespace iane_gb {

// Whether rows of nx columns take 16 lanes side by side instead of 32: where that leaves no half of a
// warp idle, on rows of up to `most` times 64. 256 x 512 rows of 64, mirror, block-wide kernel / 32 lanes / 16: 7 separable
// taps 39 / 47 / 27 us, 5 x 5 x 5 erosion 48 / 41 / 23; of 160, 78 / 86 / 64 and 78 / 72 / 56.
inline bool ring_narrow(int nx, int most)
{
	const int tiles = (nx + 63) / 64;
	return tiles % 2 == 1 && tiles <= most;
}

// Output planes per block: every chunk reads 2 r more, so as long as fills whole waves of `slots`
// resident blocks; `columns` blocks side by side. Counts of chunks of the same length are looked at once
// (one by one the loop took 15 us more of each call on 16 x 16 x 4096 voxels, whose kernel takes 18); `looked`, if
// set, is how many were.
inline int ring_chunk(long long columns, int nz, int r, long long slots, int* looked = nullptr)
{
	double best = -1.0;
	int best_zc = nz;
	for (int chunks = 1; chunks <= nz;) {
		const int zc = (nz + chunks - 1) / chunks;
		const long long blocks = columns * ((nz + zc - 1) / zc);
		const double waves = static_cast<double>(blocks) / static_cast<double>(slots);
		const double score = waves / static_cast<double>((blocks + slots - 1) / slots) * zc / (zc + 2.0 * r);
		if (looked) ++*looked;
		if (score > best + 1e-9) {
			best = score;
			best_zc = zc;
		}
		if (waves > 8.0 || zc == 1) break;
		chunks = (nz + zc - 2) / (zc - 1); // the fewest of shorter ones
	}
	return best_zc;
}

}  // namespace iane_gb
