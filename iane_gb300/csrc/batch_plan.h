// Host side of the batched Richardson-Lucy run that needs no device (plain C++: the host tests use it too).
#pragma once

#include <cstdint>
#include <sstream>
#include <string>
#include <vector>

namespace iane_gb {

// What a tuned choice was measured with: raised whenever the launch's candidates, what they mean or the
// kernel change, so that no file's choice outlives them. (2: order 1 is a queue per PSF width; lines of
// before, without a version, measured one queue in that order and may hold order 0, 62 ms where 33 are
// to be had.)
constexpr int kTuneVersion = 2;

// The batch's signature: image count, a 64-bit FNV-1a hash of every (nx, ny, kx, ky), dtype, SMs.
inline std::string tune_key(const std::vector<int>& nx, const std::vector<int>& ny, const std::vector<int>& kx,
	const std::vector<int>& ky, int sms)
{
	uint64_t h = 1469598103934665603ull;
	auto mix = [&](int v) {
		for (int b = 0; b < 4; ++b) {
			h ^= static_cast<uint64_t>((static_cast<uint32_t>(v) >> (8 * b)) & 0xffu);
			h *= 1099511628211ull;
		}
	};
	for (size_t i = 0; i < nx.size(); ++i) {
		mix(nx[i]);
		mix(ny[i]);
		mix(kx[i]);
		mix(ky[i]);
	}
	std::ostringstream k;
	k << "rl2d-batch v" << kTuneVersion << " f32 images " << nx.size() << " shapes " << std::hex << h << std::dec << " sms " << sms;
	return k.str();
}

}  // namespace iane_gb
