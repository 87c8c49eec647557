// Host side of the batched Richardson-Lucy run that needs no device (plain C++: the host tests use it too).
#pragma once

#include <algorithm>
#include <cstdint>
#include <sstream>
#include <string>
#include <vector>

namespace iane_gb {

// Tile edge of every work item (64 x 64 outputs; the body is 2 x 2 warps of 32 x 32).
constexpr int kBatchTile = 64;

// `count` consecutive 64x64 tiles of one tile row of an image: the item's shape is (64 count) x 64
// (count is 1, 2 or 4, chosen per PSF size by the autotuner).
struct alignas(16) BatchItem {
	int image;
	int x0, y0; // origin of the first tile
	int count;
	int image_tiles; // the image's 64x64 tiles (its completions per phase)
	int kx, ky;
	int reserved;
};

// Queues of one launch: at most one per PSF width (odd, 1 .. 31).
constexpr int kBatchClasses = 16;
constexpr int kBatchSmTable = 512;

// One queue: items first .. first + count - 1 of a phase, taken phases times over, and what one
// of them costs on average (any unit).
struct BatchClass {
	int first;
	int count;
	float cost;
};

// The queues of a launch and which of them the CTAs of each SM start on.
struct BatchQueues {
	int classes;
	int sms;
	int ahead; // a CTA takes its next item while it works on one (batch_ahead)
	BatchClass of[kBatchClasses];
	unsigned char start[kBatchSmTable]; // by SM id, modulo sms
};

inline int tiles_of(int n) { return (n + kBatchTile - 1) / kBatchTile; }

// Queue orders of one phase's items (the autotuner picks one per batch).
constexpr int kOrderLargestFirst = 0; // one queue, images by descending tile count
constexpr int kOrderByWidth = 1;      // a queue per PSF width, images by descending tile count
constexpr int kOrders = 2;

// Item shapes: tiles per item (along x) by PSF width, one rule per grouping level. Narrow PSFs
// do little arithmetic per tile, so their items carry the per-item queue, dependency and
// completion work over several tiles and load the taps once.
constexpr int kGroups = 4;
inline int tiles_per_item(int kx, int group)
{
	switch (group) {
	case 1: return kx <= 11 ? 2 : 1;
	case 2: return kx <= 11 ? 4 : 1;
	case 3: return kx <= 7 ? 4 : (kx <= 15 ? 2 : 1);
	default: return 1;
	}
}

// The items of one phase, queue after queue.
inline std::vector<BatchItem> make_items(const std::vector<int>& nx, const std::vector<int>& ny, const std::vector<int>& kx,
	const std::vector<int>& ky, int order, int group)
{
	const int n = static_cast<int>(nx.size());
	std::vector<int> idx(n);
	for (int i = 0; i < n; ++i) idx[i] = i;
	auto tiles = [&](int i) { return tiles_of(nx[i]) * tiles_of(ny[i]); };
	std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) {
		if (order == kOrderByWidth && kx[a] != kx[b]) return kx[a] < kx[b];
		return tiles(a) > tiles(b);
	});
	std::vector<BatchItem> items;
	for (int i : idx) {
		const int tx = tiles_of(nx[i]), ty = tiles_of(ny[i]), s = tiles_per_item(kx[i], group);
		for (int r = 0; r < ty; ++r) {
			for (int c = 0; c < tx; c += s) {
				items.push_back(BatchItem{i, c * kBatchTile, r * kBatchTile, std::min(s, tx - c), tx * ty, kx[i], ky[i], 0});
			}
		}
	}
	return items;
}

// What an item of a kx x ky PSF costs, in taps of a 64x64 tile: the taps of its 32x32 quadrants
// that touch the image, and per tile kTileOverhead for staging, hand-off and epilogue (measured
// with four CTAs per SM on 512x512 images: 2.6 SM-microseconds a tile plus 0.0187 per tap).
constexpr float kTileOverhead = 140.0f;
inline float item_cost(const BatchItem& item, int nx, int ny)
{
	const int cols = (std::min(nx, item.x0 + item.count * kBatchTile) - item.x0 + 31) / 32;
	const int rows = (std::min(ny, item.y0 + kBatchTile) - item.y0 + 31) / 32;
	return static_cast<float>(cols * rows) * 0.25f * static_cast<float>(item.kx * item.ky) +
		kTileOverhead * static_cast<float>(item.count);
}

// Whether a CTA takes its next item while it works on one. With few items per phase it holds one that an idle
// CTA could begin: 16 images of up to 300 pixels a side (273 items, 304 CTAs), 3 x 3, 0.34 -> 0.32 ms without; 16 of up
// to 700 (1243, 608) 0.55 -> 0.51; 8 of up to 1400 (2477) 0.97 with, 1.04 without.
inline bool batch_ahead(size_t items, int ctas) { return items >= 4 * static_cast<size_t>(ctas); }

// The queues of make_items' list: one for the whole batch, or one per PSF width with the SMs
// shared out in proportion to the widths' work (at least one SM each, largest remainders).
inline BatchQueues make_queues(const std::vector<BatchItem>& items, const std::vector<int>& nx, const std::vector<int>& ny,
	int order, int sms, int ctas)
{
	BatchQueues q{};
	q.ahead = batch_ahead(items.size(), ctas) ? 1 : 0;
	q.sms = std::max(1, std::min(sms, kBatchSmTable));
	double work[kBatchClasses] = {}, all = 0.0;
	for (size_t i = 0; i < items.size(); ++i) {
		const bool next = i == 0 || (order == kOrderByWidth && items[i].kx != items[i - 1].kx);
		if (next) q.of[q.classes++] = BatchClass{static_cast<int>(i), 0, 0.0f};
		++q.of[q.classes - 1].count;
		const double c = item_cost(items[i], nx[items[i].image], ny[items[i].image]);
		work[q.classes - 1] += c;
		all += c;
	}
	// as many SMs as the share gives, rounded by largest remainder; a queue whose share is
	// below one SM still gets one while there are SMs for every queue
	std::vector<int> sm(q.classes, 0);
	int left = q.sms;
	for (int c = 0; c < q.classes; ++c) {
		q.of[c].cost = static_cast<float>(work[c] / q.of[c].count);
		sm[c] = std::max(1, static_cast<int>(work[c] / all * q.sms));
		left -= sm[c];
	}
	auto short_of = [&](int c) { return work[c] / all * q.sms - sm[c]; };
	for (; left > 0 && q.classes > 0; --left) {
		int best = 0;
		for (int c = 1; c < q.classes; ++c)
			if (short_of(c) > short_of(best)) best = c;
		++sm[best];
	}
	for (; left < 0; ++left) {
		int best = -1;
		for (int c = 0; c < q.classes; ++c)
			if (sm[c] > 0 && (best < 0 || sm[c] > sm[best])) best = c;
		if (best < 0) break;
		--sm[best];
	}
	int at = 0;
	for (int c = 0; c < q.classes; ++c)
		for (int k = 0; k < sm[c] && at < q.sms; ++k) q.start[at++] = static_cast<unsigned char>(c);
	return q;
}

// CTAs per SM of a launch that is not tuned: no more than one phase has items for.
inline int default_blocks_per_sm(size_t items, int most, int sms)
{
	const long long want = (static_cast<long long>(items) + sms - 1) / sms;
	return static_cast<int>(std::max(1LL, std::min<long long>(most, want)));
}

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
