// Threads side by side in a block of the 2-D morphology kernels (plain C++: the host tests use it too).
#pragma once

namespace iane_gb {

constexpr int kPlaneThreads = 128; // of a block

// For nx x ny images, px x rows elements per thread, source rows 16-byte aligned or not, the larger
// radius r. Row ends cost a warp both ways of loading, and threads beyond them are idle: the fewer
// threads side by side, the fewer warps have either. f32 (px = 4) on aligned rows takes 8 (a warp's four
// rows of 128 bytes); elsewhere lines are shared by neighbouring threads, and it is 32 or 16 by the
// fewer elements in whole blocks, with no more than 5% between them 16 for radius 3 and 4 on rows of more
// than 256 elements (5 x 5 of a 2560 x 1920 u8 image is a microsecond faster with 32). Never more than a
// row needs, nor blocks much taller than the image. 8e6 elements, 32 -> these: f32 7 x 1 on 300 columns 46 -> 35 us (tiled kernel 40), 9 x 9 on 1300
// 60 -> 53 (58); i16 9 x 1 on 301 42 -> 34 (39); u8 9 x 9 on 2560 6% less; 0.4e6: f32 9 x 9 on 20000 rows of
// 64 26.8 -> 16.8 (17.6), i16 18.6 -> 12.4 (17.3).
inline int plane_lanes(int nx, int ny, int px, int rows, bool aligned, int r)
{
	const bool f32 = px == 4;
	auto cells = [&](int lanes) { // of whole blocks
		const int w = lanes * px, h = kPlaneThreads / lanes * rows;
		return static_cast<float>((nx + w - 1) / w * w) * static_cast<float>((ny + h - 1) / h * h);
	};
	const float c32 = cells(32), c16 = cells(16);
	int lanes = 32;
	if (c16 < 0.95f * c32 || (!f32 && r > 2 && c16 < 1.05f * c32 && nx > 256)) lanes = 16;
	// grids of a few waves: a row of blocks more can be a wave more (1171 x 512 f32 9 x 9 8.5 and 10.4 us)
	const float c = lanes == 16 ? c16 : c32, c8 = cells(8);
	if (f32 && aligned && r > 0 && c8 < (c < kPlaneThreads * 16 * 1024.0f ? 1.0f : 1.05f) * c) lanes = 8;
	while (lanes > 1 && lanes / 2 * px >= nx) lanes /= 2;
	return lanes;
}

}  // namespace iane_gb
