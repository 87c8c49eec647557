// Cube erosion and dilation of 3-D f32 volumes (radius 1, 2 or 3 along every axis): warps that march
// down z on their own; the definition stands in morphology.cu.
//
// What bounds it: memory (8 B per voxel), as long as the compare-selects (two instructions each)
// keep up. The tiled cube kernel stages every plane in shared memory cell by cell, reads it
// back one sample at a time for the x windows, stores and reads those again for the y windows,
// with two block barriers per plane. Here nothing is shared between warps and nothing is stored
// before the result:
//   * a lane owns 4 neighbouring columns and 4 rows of the warp's 128 x 4. The 4 + 2 R rows of a
//     plane, with four columns on either side, come by one TMA into a ring of the warp's own, two
//     planes ahead: no registers are tied up and no block barrier is needed. Outside the image the
//     TMA's zeros are the zero border; warps at an edge rewrite those cells for the others;
//   * the x windows of a row, then the y windows of a column, four at a time, from running
//     partial extremes (see four_windows);
//   * along z the 2 R unfinished outputs of every voxel stay in registers: a plane's result
//     completes the oldest and joins the others.
// Erosion, zero border, tiled cube kernel -> here: 384 x 384 x 256 5 x 5 x 5 131 -> 58 us (76% of the
// measured HBM rate), 7 x 7 x 7 189 -> 78; 512^3 3 x 3 x 3 302 -> 170, 5 x 5 x 5 392 -> 181 us (87%),
// 7 x 7 x 7 551 -> 252. (With the next plane's rows loaded into registers and the
// neighbours' columns by lane shuffles, two of a warp's 32 lanes without output: 124 us, the loads'
// latency exposed at three blocks per SM. With a 16-byte cp.async per lane and row: 105 us where it
// does not spill, the addresses take the registers.)
//
// The scan order is the reference's (along each axis increasing for erosion, decreasing for
// dilation, an update only on a strict compare), so that NaN and signed zeros give its bits. A
// compare and a select, both half-rate, are then 80% of what the kernel can issue (143 us). The
// one-instruction minimum skips NaN as the rule does and differs only where -0 and +0 meet; so a
// warp looks at each plane for a -0 (the lowest integer: one integer minimum per sample) and takes
// the exact form for the planes whose windows hold one.
#include "common.cuh"
#include "kernels.h"

#include <algorithm>
#include <limits>

namespace iane_gb {
namespace {

constexpr int OUT = 4;              // columns, and rows, of a lane
constexpr int COLUMNS = 32 * OUT;   // output columns of a warp
constexpr int STAGES = 3;           // planes of a warp's ring
constexpr int GROUPS = 34;          // 16-byte groups of a row there: the lanes' and one on either side
constexpr int FIXES = 64;           // cells beside the image in a warp's plane: at most 2 R x (4 + 2 R)
// bytes of a plane of the ring (TMA writes to multiples of 128)
__host__ __device__ constexpr int plane_bytes(int r) { return ((OUT + 2 * r) * GROUPS * 16 + 127) & ~127; }
__host__ __device__ constexpr int ring_bytes(int r) { return STAGES * plane_bytes(r); }
constexpr int WARPS = 4;            // warps of a block, one above the other

struct MarchArgs {
	char* dst;
	long long d_plane;
	int d_row;                // bytes; every in-plane offset fits in an int
	int nx, ny, nz;
	int border;
	int zc;                   // output planes of a block
	int dst16;                // destination rows 16-byte aligned
	int* status;
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

// Whether any of the samples is -0 in any lane: -0 has the bits of the lowest integer.
template<int ROWS, int N> __device__ __forceinline__ bool any_minus_zero(const float (&v)[ROWS][N])
{
	int low = 0;
#pragma unroll
	for (int r = 0; r < ROWS; ++r)
#pragma unroll
		for (int i = 0; i < N; ++i) low = min(low, __float_as_int(v[r][i]));
	return __any_sync(0xffffffffu, low == std::numeric_limits<int>::min());
}

// w: a row's columns with R on either side
template<bool DILATE, bool FAST, int R, int ROWS>
__device__ __forceinline__ void x_windows(const float (&w)[ROWS][OUT + 2 * R], float (&h)[ROWS][OUT])
{
#pragma unroll
	for (int r = 0; r < ROWS; ++r) four_windows<DILATE, FAST, R>(w[r], h[r]);
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

template<bool DILATE, int R>
__global__ void __launch_bounds__(32 * WARPS, R == 3 ? 2 : R == 2 ? 3 : 4)
	morph_march_kernel(const __grid_constant__ CUtensorMap map, const MarchArgs a)
{
	constexpr int ROWS = OUT + 2 * R;
	extern __shared__ __align__(128) unsigned char smem[];
	const int lane = threadIdx.x, warp = threadIdx.y;
	unsigned char* ring = smem + warp * ring_bytes(R);
	uint64_t* bars = reinterpret_cast<uint64_t*>(smem + WARPS * ring_bytes(R)) + warp * STAGES;
	const int xw = blockIdx.x * COLUMNS; // the warp's first column
	const int x = xw + OUT * lane;
	const int y0 = (blockIdx.y * WARPS + warp) * OUT;
	const int z0 = blockIdx.z * a.zc, z1 = min(a.nz, z0 + a.zc);
	if (y0 >= a.ny) return;
	if (lane == 0) {
		for (int k = 0; k < STAGES; ++k) mbar_init(&bars[k], 1);
		fence_barrier_init();
	}
	__syncwarp();
	const bool whole = x + OUT <= a.nx;
	const bool mapped = a.border != IANE_GB_BORDER_ZERO;
	// clamp and mirror: the warp's planes reach over an edge of the image
	const bool edge_x = mapped && (xw == 0 || xw + COLUMNS + R > a.nx);
	const bool edge_y = mapped && (y0 < R || y0 + OUT + R > a.ny);

	auto issue = [&](int z, int slot) { // lane 0
		int zi = 0;
		if (!map_coord(z, a.nz, a.border, zi)) zi = z; // the zero border's plane: zeros
		// order the warp's reads and edge writes of the slot before the copy into it
		asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
		mbar_arrive_expect_tx(&bars[slot], ROWS * GROUPS * 16);
		tma_load_3d(ring + slot * plane_bytes(R), &map, xw - OUT, y0 - R, zi, &bars[slot]);
	};
	// clamp and mirror: the cells outside the image that windows of stored outputs reach, from where
	// the rule takes them (within the warp's rows and columns, as the image is 16 or more of each).
	// Found once, the same in every plane: cells beside the rows (cell << 16 | source), then whole rows
	int* const fixes = reinterpret_cast<int*>(smem + WARPS * (ring_bytes(R) + STAGES * 8)) + warp * (FIXES + 16);
	int* const row_from = fixes + FIXES;
	unsigned fix_rows = 0;
	if (edge_x) {
		for (int i = lane; i < FIXES; i += 32) {
			const int r = i / (2 * R), j = i - r * 2 * R;
			const int c = j < R ? -R + j : a.nx + j - R; // column
			int from = 0;
			map_coord(c, a.nx, a.border, from);
			const int to_at = c - xw + OUT, from_at = from - xw + OUT;
			const bool here = r < ROWS && to_at >= 0 && to_at < 4 * GROUPS && from_at >= 0 && from_at < 4 * GROUPS;
			fixes[i] = here ? (r * 4 * GROUPS + to_at) << 16 | (r * 4 * GROUPS + from_at) : -1;
		}
	}
	if (edge_y) {
		for (int r = 0; r < ROWS; ++r) {
			const int y = y0 - R + r;
			if ((y >= 0 && y < a.ny) || y >= a.ny + R) continue;
			int from = 0;
			map_coord(y, a.ny, a.border, from);
			const int from_r = from - (y0 - R);
			if (from_r < 0 || from_r >= ROWS) continue;
			fix_rows |= 1u << r;
			if (lane == 0) row_from[r] = from_r;
		}
	}
	__syncwarp();
	auto fix = [&](float* plane) {
		if (edge_x) {
#pragma unroll
			for (int i = 0; i < 2 * R * ROWS; i += 32) {
				const int e = fixes[i + lane];
				if (e >= 0) plane[e >> 16] = plane[e & 0xffff];
			}
			__syncwarp();
		}
		if (edge_y) {
			float4* rows = reinterpret_cast<float4*>(plane);
			for (unsigned left = fix_rows; left; left &= left - 1) {
				const int r = __ffs(left) - 1;
				float4* to = rows + r * GROUPS;
				const float4* from = rows + row_from[r] * GROUPS;
				to[lane] = from[lane];
				if (lane < GROUPS - 32) to[32 + lane] = from[32 + lane];
			}
			__syncwarp();
		}
	};

	// unfinished outputs: pending[k] has seen its first 2 R - k planes
	float pending[2 * R][OUT][OUT];
	const float start = DILATE ? -std::numeric_limits<float>::infinity() : std::numeric_limits<float>::infinity();
#pragma unroll
	for (int k = 0; k < 2 * R; ++k)
#pragma unroll
		for (int j = 0; j < OUT; ++j)
#pragma unroll
			for (int i = 0; i < OUT; ++i) pending[k][j][i] = start;

	if (lane == 0) {
		for (int k = 0; k < STAGES - 1 && z0 - R + k < z1 + R; ++k) issue(z0 - R + k, k);
	}
	int since = 2 * R; // planes since one that holds a -0
	int slot = 0;
	uint32_t parity = 0;
	bool ok = true;
	for (int z = z0 - R; z < z1 + R; ++z) {
		__syncwarp(); // every lane has read the plane before this one: its slot takes the next copy
		if (lane == 0 && z + STAGES - 1 < z1 + R) issue(z + STAGES - 1, slot == 0 ? STAGES - 1 : slot - 1);
		if (ok && !mbar_wait_bounded(&bars[slot], parity)) {
			ok = false;
			report_device_status(a.status, IANE_GB_DEVICE_TIMEOUT);
		}
		__syncwarp();
		unsigned char* plane = ring + slot * plane_bytes(R);
		if (edge_x || edge_y) fix(reinterpret_cast<float*>(plane));
		float w[ROWS][OUT + 2 * R];
		const float4* from = reinterpret_cast<const float4*>(plane) + lane;
		if (++slot == STAGES) {
			slot = 0;
			parity ^= 1u;
		}
#pragma unroll
		for (int r = 0; r < ROWS; ++r) {
			const float4 q = from[r * GROUPS + 1];
			w[r][R] = q.x;
			w[r][R + 1] = q.y;
			w[r][R + 2] = q.z;
			w[r][R + 3] = q.w;
			const float* beside = reinterpret_cast<const float*>(from + r * GROUPS + 1);
			if constexpr (R == 2) {
				const float2 lo = *reinterpret_cast<const float2*>(beside - 2), hi = *reinterpret_cast<const float2*>(beside + 4);
				w[r][0] = lo.x;
				w[r][1] = lo.y;
				w[r][6] = hi.x;
				w[r][7] = hi.y;
			} else {
#pragma unroll
				for (int j = 0; j < R; ++j) {
					w[r][j] = beside[j - R];
					w[r][R + OUT + j] = beside[OUT + j];
				}
			}
		}
		float h[ROWS][OUT], m[OUT][OUT];
		const bool minus = any_minus_zero(w);
		since = minus ? 0 : since + 1;
		if (minus) {
			x_windows<DILATE, false, R>(w, h);
			y_windows<DILATE, false, R>(h, m);
		} else {
			x_windows<DILATE, true, R>(w, h);
			y_windows<DILATE, true, R>(h, m);
		}
		if (since <= 2 * R) {
			z_windows<DILATE, false, R>(pending, m);
		} else {
			z_windows<DILATE, true, R>(pending, m);
		}
		const int zo = z - R; // the output plane that this plane completed
		if (zo >= z0) {
			char* plane = a.dst + zo * a.d_plane;
#pragma unroll
			for (int j = 0; j < OUT; ++j) {
				if (y0 + j >= a.ny) break;
				float* row = reinterpret_cast<float*>(plane + (y0 + j) * a.d_row) + x;
				if (a.dst16 && whole) {
					*reinterpret_cast<float4*>(row) = make_float4(m[j][0], m[j][1], m[j][2], m[j][3]);
				} else {
#pragma unroll
					for (int i = 0; i < OUT; ++i) {
						if (x + i < a.nx) row[i] = m[j][i];
					}
				}
			}
		}
	}
}

template<bool DILATE, int R>
int launch(const CUtensorMap& map, const MarchArgs& a, dim3 grid, cudaStream_t st)
{
	constexpr size_t smem = static_cast<size_t>(WARPS) * (ring_bytes(R) + STAGES * 8 + (FIXES + 16) * 4);
	auto kernel = morph_march_kernel<DILATE, R>;
	IANE_GB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
		"morphology: set shared memory size");
	kernel<<<grid, dim3(32, WARPS), smem, st>>>(map, a);
	IANE_GB_CUDA(cudaGetLastError(), "morphology: launch");
	return IANE_GB_OK;
}

template<bool DILATE>
int launch_radius(const CUtensorMap& map, const MarchArgs& a, int r, dim3 grid, cudaStream_t st)
{
	return r == 1 ? launch<DILATE, 1>(map, a, grid, st) : r == 2 ? launch<DILATE, 2>(map, a, grid, st)
		: launch<DILATE, 3>(map, a, grid, st);
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
	// rows and planes that TMA can address: 16-byte aligned, one after the other
	if (s.dtype != IANE_GB_F32 || r[0] != r[1] || r[1] != r[2] || r[0] < 1 || r[0] > 3 || !rows_aligned16(s) ||
	    s.stride[1] < 4LL * s.ext[0] || (s.ext[2] > 1 && s.stride[2] < s.stride[1] * s.ext[1]) || d.stride[0] != 4 ||
	    s.ext[0] < 16 || s.ext[1] < 16 || !plane_fits(d)) {
		return IANE_GB_UNSUPPORTED;
	}
	// 7 x 7 x 7 on the smallest volumes stays with the tiled kernel, whose blocks are more and shorter
	// (32 x 64 x 64, mirror: 10.4 us there, 11.5 here; 20 x 300 x 400: 30.4 and 19.9)
	if (r[0] == 3 && element_count(s) < (1LL << 18)) return IANE_GB_UNSUPPORTED;
	MarchArgs a{};
	a.status = device_status_ptr();
	if (!a.status) return IANE_GB_CUDA_ERROR;
	a.dst = d.ptr;
	a.d_plane = d.stride[2];
	a.d_row = static_cast<int>(d.stride[1]);
	a.nx = s.ext[0];
	a.ny = s.ext[1];
	a.nz = s.ext[2];
	a.border = border;
	a.dst16 = rows_aligned16(d) ? 1 : 0;
	// planes per block: every chunk reads 2 R more, so as long as fills whole waves of resident blocks
	const dim3 tiles((a.nx + COLUMNS - 1) / COLUMNS, (a.ny + OUT * WARPS - 1) / (OUT * WARPS));
	const long long columns = static_cast<long long>(tiles.x) * tiles.y;
	const long long slots = static_cast<long long>(r[0] == 3 ? 2 : r[0] == 2 ? 3 : 4) * device_sm_count();
	double best = -1.0;
	for (int chunks = 1; chunks <= a.nz; ++chunks) {
		const int zc = (a.nz + chunks - 1) / chunks;
		const long long blocks = columns * ((a.nz + zc - 1) / zc);
		const double waves = static_cast<double>(blocks) / static_cast<double>(slots);
		const double fill = waves / static_cast<double>((blocks + slots - 1) / slots);
		const double score = fill * zc / (zc + 2.0 * r[0]);
		if (score > best + 1e-9) {
			best = score;
			a.zc = zc;
		}
		if (waves > 8.0) break;
	}
	CUtensorMap map{};
	const int status = encode_tensor_map_f32(&map, s.ptr, a.nx, a.ny, a.nz, s.stride[1],
		a.nz > 1 ? s.stride[2] : s.stride[1] * a.ny, 4 * GROUPS, OUT + 2 * r[0]);
	if (status) return status;
	const dim3 grid(tiles.x, tiles.y, (a.nz + a.zc - 1) / a.zc);
	return dilate ? launch_radius<true>(map, a, r[0], grid, st) : launch_radius<false>(map, a, r[0], grid, st);
}

}  // namespace iane_gb
