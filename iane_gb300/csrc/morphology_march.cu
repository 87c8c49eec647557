// Cube erosion and dilation of 3-D f32 volumes (radius 1, 2 or 3 along every axis): warps that march
// down z on their own; the definition stands in morphology.cu.
//
// What bounds it: memory (8 B per voxel), as long as the compare-selects (two instructions each)
// keep up. The tiled cube kernel stages every plane in shared memory cell by cell, reads it
// back one sample at a time for the x windows, stores and reads those again for the y windows,
// with two block barriers per plane. Here nothing is shared between warps and nothing is stored
// before the result:
//   * a lane owns 4 neighbouring columns and 4 rows of the warp's 128 x 4, or 64 x 8 (ring_narrow).
//     The planes come by TMA into a ring of the warp's own (warp_ring.cuh): no registers are tied up and no block barrier
//     is needed;
//   * the x windows of a row, then the y windows of a column, four at a time, from running
//     partial extremes (see four_windows);
//   * along z the 2 R unfinished outputs of every voxel stay in registers: a plane's result
//     completes the oldest and joins the others.
// Erosion, zero border, tiled cube kernel -> here: 384 x 384 x 256 3 x 3 x 3 98 -> 53 us, 5 x 5 x 5
// 131 -> 61 (73% of the measured HBM rate), 7 x 7 x 7 189 -> 83; 512^3 3 x 3 x 3 302 -> 167 us (95%),
// 5 x 5 x 5 392 -> 190, 7 x 7 x 7 551 -> 265; mirror up to a sixth more. (With the next plane's rows
// loaded into registers and the neighbours' columns by lane shuffles, two of a warp's 32 lanes without
// output: 124 us, the loads' latency exposed at three blocks per SM. With a 16-byte cp.async per lane
// and row: 105 us where it does not spill, the addresses take the registers.)
//
// The scan order is the reference's (along each axis increasing for erosion, decreasing for
// dilation, an update only on a strict compare), so that NaN and signed zeros give its bits. A
// compare and a select, both half-rate, are then 80% of what the kernel can issue (143 us). The
// one-instruction minimum skips NaN as the rule does and differs only where -0 and +0 meet; so a
// warp looks at each plane for a -0 (the lowest integer: one integer minimum per sample) and takes
// the exact form for the planes whose windows hold one.
#include "kernels.h"
#include "warp_ring.cuh"

#include <algorithm>
#include <limits>

namespace iane_gb {
namespace {

constexpr int OUT = kRingOut;       // columns, and rows, of a lane
constexpr int WARPS = 4;            // warps of a block, one above the other

struct MarchArgs {
	RingArgs in;
	char* dst;
	long long d_plane;
	int d_row;                // bytes; every in-plane offset fits in an int
	int zc;                   // output planes of a block
	int dst16;                // destination rows 16-byte aligned
};

// The extreme of `first`, then `then`, in scan order: `then` replaces it on a strict compare. FAST:
// the one-instruction minimum or maximum, which differs only in which of -0 and +0 it keeps.
template<bool DILATE, bool FAST> __device__ __forceinline__ float join(float first, float then)
{
	if constexpr (FAST) return DILATE ? fmaxf(first, then) : fminf(first, then);
	return (DILATE ? then > first : then < first) ? then : first;
}

// Four neighbouring windows of 2 R + 1 from OUT + 2 R samples (NaN among them), in the reference's
// order. For 2 R >= OUT every window holds samples OUT - 1 and OUT: its part up to OUT - 1 and its
// part from OUT are running extremes shared by the four (the update rule is associative over
// consecutive runs of the scan). Erosion scans upwards: the lower part extended downwards keeps
// the new sample on ties, the upper one extended upwards keeps the old; dilation mirrors this.
template<bool DILATE, bool FAST, int R>
__device__ __forceinline__ void four_windows(const float (&v)[OUT + 2 * R], float (&m)[OUT])
{
	const float start = DILATE ? -std::numeric_limits<float>::infinity() : std::numeric_limits<float>::infinity();
	if constexpr (2 * R >= OUT) {
		float part[OUT];
		float run = start;
#pragma unroll
		for (int k = OUT - 1; k >= 0; --k) {
			if constexpr (FAST) {
				run = join<DILATE, true>(run, v[k]);
			} else if (DILATE ? v[k] > run : v[k] <= run) {
				run = v[k];
			}
			part[k] = run;
		}
		float edge = start;
#pragma unroll
		for (int j = OUT; j < OUT + 2 * R; ++j) {
			if constexpr (FAST) {
				edge = join<DILATE, true>(edge, v[j]);
			} else if (DILATE ? v[j] >= edge : v[j] < edge) {
				edge = v[j];
			}
			const int k = j - 2 * R;
			if (k >= 0) m[k] = DILATE ? join<true, FAST>(edge, part[k]) : join<false, FAST>(part[k], edge);
		}
	} else {
#pragma unroll
		for (int k = 0; k < OUT; ++k) {
			float run = start;
#pragma unroll
			for (int o = 0; o <= 2 * R; ++o) run = join<DILATE, FAST>(run, v[k + (DILATE ? 2 * R - o : o)]);
			m[k] = run;
		}
	}
}

// The x windows of a plane's rows. Returns whether one of the samples is -0 (the lowest integer by
// its bits) in any lane.
template<bool DILATE, bool FAST, int R, bool EDGE, class Ring>
__device__ __forceinline__ bool x_windows(const Ring& ring, const float4* plane, float (&h)[OUT + 2 * R][OUT])
{
	int low = 0;
#pragma unroll
	for (int r = 0; r < OUT + 2 * R; ++r) {
		float w[OUT + 2 * R];
		ring.template read<EDGE>(plane, r, w);
#pragma unroll
		for (int i = 0; i < OUT + 2 * R; ++i) low = min(low, __float_as_int(w[i]));
		four_windows<DILATE, FAST, R>(w, h[r]);
	}
	return __any_sync(0xffffffffu, low == std::numeric_limits<int>::min());
}

template<bool DILATE, bool FAST, int R, int ROWS>
__device__ __forceinline__ void y_windows(const float (&h)[ROWS][OUT], float (&m)[OUT][OUT]) // m: [row][column]
{
#pragma unroll
	for (int i = 0; i < OUT; ++i) {
		float col[ROWS], out[OUT];
#pragma unroll
		for (int r = 0; r < ROWS; ++r) col[r] = h[r][i];
		four_windows<DILATE, FAST, R>(col, out);
#pragma unroll
		for (int j = 0; j < OUT; ++j) m[j][i] = out[j];
	}
}

// The plane completes the oldest output (left in m) and joins the others: erosion scans it after
// what they have seen, dilation before.
template<bool DILATE, bool FAST, int R>
__device__ __forceinline__ void z_windows(float (&pending)[2 * R][OUT][OUT], float (&m)[OUT][OUT])
{
#pragma unroll
	for (int j = 0; j < OUT; ++j) {
#pragma unroll
		for (int i = 0; i < OUT; ++i) {
			const float p = m[j][i];
			m[j][i] = DILATE ? join<true, FAST>(p, pending[0][j][i]) : join<false, FAST>(pending[0][j][i], p);
#pragma unroll
			for (int k = 0; k + 1 < 2 * R; ++k) {
				const float seen = pending[k + 1][j][i];
				pending[k][j][i] = DILATE ? join<true, FAST>(p, seen) : join<false, FAST>(seen, p);
			}
			pending[2 * R - 1][j][i] = p;
		}
	}
}

template<bool DILATE, int R, int LANES>
__global__ void __launch_bounds__(32 * WARPS, R == 3 ? 2 : R == 2 ? 3 : 4)
	morph_march_kernel(const __grid_constant__ CUtensorMap map, const MarchArgs a)
{
	using Ring = WarpRing<R, LANES>;
	constexpr int ROWS = OUT + 2 * R;
	extern __shared__ __align__(128) unsigned char smem[];
	const int warp = threadIdx.y, warps = LANES == 32 ? WARPS : blockDim.y;
	const int nx = a.in.nx, ny = a.in.ny;
	const int xw = blockIdx.x * Ring::COLUMNS, yw = (blockIdx.y * warps + warp) * Ring::OUT_ROWS; // the warp's first
	const int x = xw + Ring::column(), y0 = yw + Ring::row();
	const int z0 = blockIdx.z * a.zc, z1 = min(a.in.nz, z0 + a.zc);
	if (yw >= ny) return;
	const bool whole = x + OUT <= nx;
	Ring ring;
	ring.begin(smem, warps, warp, &map, a.in, xw, yw, z0 - R, z1 + R);

	// unfinished outputs: pending[k] has seen its first 2 R - k planes
	float pending[2 * R][OUT][OUT];
	const float start = DILATE ? -std::numeric_limits<float>::infinity() : std::numeric_limits<float>::infinity();
#pragma unroll
	for (int k = 0; k < 2 * R; ++k)
#pragma unroll
		for (int j = 0; j < OUT; ++j)
#pragma unroll
			for (int i = 0; i < OUT; ++i) pending[k][j][i] = start;

	int since = 2 * R; // planes since one that holds a -0
	for (int z = z0 - R; z < z1 + R; ++z) {
		const float4* plane = ring.plane(&map, a.in, z);
		float h[ROWS][OUT], m[OUT][OUT];
		bool minus = ring.edge ? x_windows<DILATE, true, R, true>(ring, plane, h) : x_windows<DILATE, true, R, false>(ring, plane, h);
		since = minus ? 0 : since + 1;
		if (minus) {
			if (ring.edge) {
				x_windows<DILATE, false, R, true>(ring, plane, h);
			} else {
				x_windows<DILATE, false, R, false>(ring, plane, h);
			}
			y_windows<DILATE, false, R>(h, m);
		} else {
			y_windows<DILATE, true, R>(h, m);
		}
		if (z + 1 < z1 + R) ring.prepare(a.in);
		if (since <= 2 * R) {
			z_windows<DILATE, false, R>(pending, m);
		} else {
			z_windows<DILATE, true, R>(pending, m);
		}
		const int zo = z - R; // the output plane that this plane completed
		if (zo >= z0) {
			char* out = a.dst + zo * a.d_plane;
#pragma unroll
			for (int j = 0; j < OUT; ++j) {
				if (y0 + j >= ny) break;
				float* row = reinterpret_cast<float*>(out + (y0 + j) * a.d_row) + x;
				if (a.dst16 && whole) {
					*reinterpret_cast<float4*>(row) = make_float4(m[j][0], m[j][1], m[j][2], m[j][3]);
				} else {
#pragma unroll
					for (int i = 0; i < OUT; ++i) {
						if (x + i < nx) row[i] = m[j][i];
					}
				}
			}
		}
	}
}

template<bool DILATE, int R, int LANES>
int launch_lanes(const DevView& s, MarchArgs a, cudaStream_t st)
{
	using Ring = WarpRing<R, LANES>;
	const int warps = ring_warps<Ring>(a.in, WARPS);
	const size_t smem = Ring::bytes(warps);
	auto kernel = morph_march_kernel<DILATE, R, LANES>;
	IANE_GB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Ring::bytes(WARPS))),
		"morphology: set shared memory size"); // the most, as other threads may launch in between
	CUtensorMap map{};
	const int status = ring_map<R, LANES>(&map, s);
	if (status) return status;
	const dim3 tiles = ring_tiles<Ring>(a.in, warps);
	a.zc = ring_chunk(static_cast<long long>(tiles.x) * tiles.y, a.in.nz, R,
		static_cast<long long>((R == 3 ? 2 : R == 2 ? 3 : 4) * WARPS / warps) * device_sm_count());
	kernel<<<dim3(tiles.x, tiles.y, (a.in.nz + a.zc - 1) / a.zc), dim3(32, warps), smem, st>>>(map, a);
	IANE_GB_CUDA(cudaGetLastError(), "morphology: launch");
	return IANE_GB_OK;
}

template<bool DILATE, int R>
int launch(const DevView& s, const MarchArgs& a, cudaStream_t st)
{
	return ring_narrow(a.in.nx, 1 << 30) ? launch_lanes<DILATE, R, 16>(s, a, st) : launch_lanes<DILATE, R, 32>(s, a, st);
}

template<bool DILATE>
int launch_radius(const DevView& s, const MarchArgs& a, int r, cudaStream_t st)
{
	return r == 1 ? launch<DILATE, 1>(s, a, st) : r == 2 ? launch<DILATE, 2>(s, a, st) : launch<DILATE, 3>(s, a, st);
}

// Whether every in-plane byte offset of the view fits in an int.
bool plane_fits(const DevView& v)
{
	const long long row = v.stride[1] < 0 ? -v.stride[1] : v.stride[1];
	return row * std::max(0, v.ext[1] - 1) + 4LL * v.ext[0] <= std::numeric_limits<int>::max();
}

}  // namespace

int launch_morph_march(const DevView& s, const DevView& d, const int* r, bool dilate, int border, cudaStream_t st)
{
	if (!ring_supported(s) || r[0] != r[1] || r[1] != r[2] || r[0] < 1 || r[0] > 3 || d.stride[0] != 4 || !plane_fits(d)) {
		return IANE_GB_UNSUPPORTED;
	}
	// 7 x 7 x 7 on the smallest volumes stays with the tiled kernel, whose blocks are more and shorter
	// (32 x 64 x 64, mirror: 10.4 us there, 11.5 here; 20 x 300 x 400: 30.4 and 19.9)
	if (r[0] == 3 && element_count(s) < (1LL << 18)) return IANE_GB_UNSUPPORTED;
	MarchArgs a{};
	a.in = RingArgs{s.ext[0], s.ext[1], s.ext[2], border, device_status_ptr()};
	if (!a.in.status) return IANE_GB_CUDA_ERROR;
	a.dst = d.ptr;
	a.d_plane = d.stride[2];
	a.d_row = static_cast<int>(d.stride[1]);
	a.dst16 = rows_aligned16(d) ? 1 : 0;
	return dilate ? launch_radius<true>(s, a, r[0], st) : launch_radius<false>(s, a, r[0], st);
}

}  // namespace iane_gb
