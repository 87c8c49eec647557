// A warp's own ring of input planes, for kernels whose warps march down z on their own (no block
// barrier). A lane has 4 columns and 4 rows; 32 lanes side by side make a warp's 128 x 4, or 16, two
// such rows of them one above the other, its 64 x 8. A plane is the warp's rows and R more on either side, its
// columns and four more on either side: one TMA per plane, two planes ahead of the one in use. Outside the image the TMA's zeros are the zero border. For clamp and
// mirror a warp at an edge reads other rows in the place of those outside, and a lane at a row's end
// takes the columns beyond it from its own four: a few selects. (Rewriting those cells in shared
// memory after every copy is a chain of latencies that the edge warps' few neighbours do not hide:
// 512^3, 7 separable taps, mirror 275 us against 230 with zeros.) Only rows that end inside a lane's
// four columns are completed in shared memory.
#pragma once

#include "common.cuh"
#include "ring_chunk.h"

namespace iane_gb {

constexpr int kRingOut = 4;                 // columns, and rows, of a lane
constexpr int kRingStages = 3;
constexpr int kRingFixes = 64;              // cells beyond the rows' ends in a plane: at most R x (8 + 2 R), R <= 4

// What the LANES side by side make of a warp.
template<int R, int SIDE>
struct RingShape {
	static_assert(SIDE == 32 || SIDE == 16, "");
	static constexpr int LANES = SIDE;
	static constexpr int COLUMNS = LANES * kRingOut;
	static constexpr int OUT_ROWS = 32 / LANES * kRingOut; // output rows
	static constexpr int ROWS = OUT_ROWS + 2 * R;          // of a plane
	static constexpr int GROUPS = LANES + 2;               // 16-byte groups of a row
	// of this thread's lane: its group and first row, and the group at which row 0 of its window begins
	static __device__ __forceinline__ int column() { return kRingOut * (LANES == 32 ? threadIdx.x : threadIdx.x & (LANES - 1)); }
	static __device__ __forceinline__ int row() { return LANES == 32 ? 0 : kRingOut * ((threadIdx.x & 31) / LANES); }
	static __device__ __forceinline__ int own() { return row() * GROUPS + (threadIdx.x & (LANES - 1)) + 1; }
};

// What a launch's warps share.
struct RingArgs {
	int nx, ny, nz; // the image, 16 or more along x and y
	int border;
	int* status;
};

// The four columns at `at` with R on either side.
template<int R> __device__ __forceinline__ void ring_row(const float4* at, float (&w)[kRingOut + 2 * R])
{
	const float4 q = at[0];
	w[R] = q.x;
	w[R + 1] = q.y;
	w[R + 2] = q.z;
	w[R + 3] = q.w;
	const float* beside = reinterpret_cast<const float*>(at);
	if constexpr (R == 2) {
		const float2 lo = *reinterpret_cast<const float2*>(beside - 2), hi = *reinterpret_cast<const float2*>(beside + 4);
		w[0] = lo.x;
		w[1] = lo.y;
		w[6] = hi.x;
		w[7] = hi.y;
	} else if constexpr (R >= 3) {
		const float4 lo = at[-1], hi = at[1];
		const float l[4] = {lo.x, lo.y, lo.z, lo.w}, h[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
		for (int j = 0; j < R; ++j) {
			w[j] = l[4 - R + j];
			w[R + kRingOut + j] = h[j];
		}
	} else {
		w[0] = beside[-1];
		w[R + kRingOut] = beside[kRingOut];
	}
}

template<int R, int LANES>
struct WarpRing : RingShape<R, LANES> {
	using Source = CUtensorMap;
	using S = RingShape<R, LANES>;
	static constexpr int WINDOW = kRingOut + 2 * R; // rows that a lane reads
	static constexpr int PLANE = (S::ROWS * S::GROUPS * 16 + 127) & ~127; // bytes; TMA writes to multiples of 128
	static constexpr int RING = kRingStages * PLANE;
	// shared memory of a block of `warps` warps
	static constexpr size_t bytes(int warps)
	{
		return static_cast<size_t>(warps) * (RING + kRingStages * 8 + kRingFixes * 4);
	}

	unsigned char* ring;
	uint64_t* bars;
	int* fixes;             // ragged rows: cell << 16 | source, or -1
	unsigned long long from; // edge: four bits per row of the lane's window, the one to read in its place
	int x0, y0, z1;
	int slot;
	uint32_t parity;
	bool edge;              // clamp or mirror, and the planes reach over an edge of the image
	bool ragged;            // and the rows end inside a group of four columns
	bool left, right;       // this lane's neighbours on that side lie outside
	bool clamp, ok;

	// Warp `warp` of `warps` begins at columns from x0, rows from y0 and input plane z, and will take
	// the planes before z_end. All lanes.
	__device__ __forceinline__ void begin(unsigned char* smem, int warps, int warp, const CUtensorMap* map, const RingArgs& a,
		int x, int y, int z, int z_end)
	{
		const int lane = threadIdx.x & 31;
		ring = smem + warp * RING;
		bars = reinterpret_cast<uint64_t*>(smem + warps * RING) + warp * kRingStages;
		fixes = reinterpret_cast<int*>(smem + warps * (RING + kRingStages * 8)) + warp * kRingFixes;
		x0 = x;
		y0 = y;
		z1 = z_end;
		slot = 0;
		parity = 0;
		ok = true;
		const bool mapped = a.border != IANE_GB_BORDER_ZERO;
		const bool edge_x = mapped && (x0 == 0 || x0 + S::COLUMNS + R > a.nx);
		const bool edge_y = mapped && (y0 < R || y0 + S::OUT_ROWS + R > a.ny);
		edge = edge_x || edge_y;
		clamp = a.border == IANE_GB_BORDER_CLAMP;
		ragged = edge_x && a.nx % kRingOut != 0 && x0 + S::COLUMNS + R > a.nx;
		left = mapped && x0 + S::column() == 0;
		right = mapped && !ragged && x0 + S::column() + kRingOut == a.nx;
		if (lane == 0) {
			for (int k = 0; k < kRingStages; ++k) mbar_init(&bars[k], 1);
			fence_barrier_init();
		}
		from = 0;
		for (int r = 0; r < WINDOW; ++r) {
			int row = y0 + S::row() - R + r, to = r;
			// rows that no stored output reads stay
			if (mapped && (row < 0 || row >= a.ny) && row < a.ny + R) {
				int yi = 0;
				map_coord(row, a.ny, a.border, yi);
				to = yi - (y0 + S::row() - R); // within the window, as the image has 16 or more
				to = to < 0 ? 0 : to >= WINDOW ? WINDOW - 1 : to;
			}
			from |= static_cast<unsigned long long>(to) << (4 * r);
		}
		if (ragged) {
			for (int i = lane; i < kRingFixes; i += 32) {
				const int r = i / R, c = a.nx + i - r * R; // column
				int xi = 0;
				map_coord(c, a.nx, a.border, xi);
				const int to_at = c - x0 + kRingOut, from_at = xi - x0 + kRingOut;
				const bool here = r < S::ROWS && to_at < 4 * S::GROUPS && from_at >= 0;
				fixes[i] = here ? (r * 4 * S::GROUPS + to_at) << 16 | (r * 4 * S::GROUPS + from_at) : -1;
			}
		}
		__syncwarp();
		if (lane == 0) {
			for (int k = 0; k < kRingStages - 1 && z + k < z1; ++k) issue(map, a, z + k, k);
		}
		prepare(a);
	}

	// Lane 0: the copy of plane z into slot `to`.
	__device__ __forceinline__ void issue(const CUtensorMap* map, const RingArgs& a, int z, int to)
	{
		int zi = 0;
		if (!map_coord(z, a.nz, a.border, zi)) zi = z; // the zero border's plane: zeros
		// order the warp's reads and edge writes of the slot before the copy into it
		asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
		mbar_arrive_expect_tx(&bars[to], S::ROWS * S::GROUPS * 16);
		tma_load_3d(ring + to * PLANE, map, x0 - kRingOut, y0 - R, zi, &bars[to]);
	}

	// Plane z, prepared, for row(). The warp is done with the plane before it, whose slot takes another
	// copy. All lanes.
	__device__ __forceinline__ const float4* plane(const CUtensorMap* map, const RingArgs& a, int z)
	{
		__syncwarp();
		if ((threadIdx.x & 31) == 0 && z + kRingStages - 1 < z1) {
			issue(map, a, z + kRingStages - 1, slot == 0 ? kRingStages - 1 : slot - 1);
		}
		const float4* rows = reinterpret_cast<const float4*>(ring + slot * PLANE);
		if (++slot == kRingStages) {
			slot = 0;
			parity ^= 1u;
		}
		return rows;
	}

	// Wait for the next plane to be taken and complete its ragged rows. All lanes.
	__device__ __forceinline__ void prepare(const RingArgs& a)
	{
		if (ok && !mbar_wait_bounded(&bars[slot], parity)) {
			ok = false;
			report_device_status(a.status, IANE_GB_DEVICE_TIMEOUT);
		}
		if (ragged) {
			float* cells = reinterpret_cast<float*>(ring + slot * PLANE);
#pragma unroll
			for (int i = 0; i < R * S::ROWS; i += 32) {
				const int e = fixes[i + (threadIdx.x & 31)];
				if (e >= 0) cells[e >> 16] = cells[e & 0xffff];
			}
		}
	}

	// Row r of the lane's window: its columns with R on either side, from plane(). EDGE: for warps with `edge`.
	template<bool EDGE> __device__ __forceinline__ void read(const float4* rows, int r, float (&w)[kRingOut + 2 * R]) const
	{
		const float4* at = rows + (EDGE ? static_cast<int>(from >> (4 * r) & 15u) : r) * S::GROUPS + S::own();
		ring_row<R>(at, w);
		if constexpr (EDGE) {
			// columns -1 - j and nx + j are columns j and nx - 1 - j under mirror
#pragma unroll
			for (int j = 0; j < R; ++j) {
				const float l = clamp ? w[R] : w[R + j], h = clamp ? w[R + kRingOut - 1] : w[R + kRingOut - 1 - j];
				w[R - 1 - j] = left ? l : w[R - 1 - j];
				w[R + kRingOut + j] = right ? h : w[R + kRingOut + j];
			}
		}
	}
};

// The same for rows that TMA cannot address: 4-byte cp.async, lane by lane along each row, from the columns and
// rows that the border rule names, so that no edge is left to the reader. (253 x 181 x 60, 7 separable
// taps, mirror: 23 us; the block-wide kernel, which maps every cell of a plane on its own, 63.)
struct CopySource {
	const char* src; // f32, contiguous along x; strides in bytes
	long long s_row, s_plane;
};

template<int R, int LANES>
struct CopyRing : RingShape<R, LANES> {
	using Source = CopySource;
	using S = RingShape<R, LANES>;
	static constexpr int PLANE = S::ROWS * S::GROUPS * 16;
	static constexpr int COPIES = (4 * S::GROUPS + 31) / 32; // of a lane per row
	static constexpr bool SPARE = S::ROWS < 16; // 15 names no row and stands for one that is not there
	static constexpr size_t bytes(int warps) { return static_cast<size_t>(warps) * (kRingStages * PLANE + 32 * COPIES * 4); }
	static constexpr bool edge = false;

	unsigned char* ring;
	int* columns;            // the source column of each, or -1
	unsigned long long from; // four bits per row, the row to read in its place
	uint32_t rows_in;        // without SPARE: a bit per row that is there
	int y0, z1;
	int slot;

	__device__ __forceinline__ void begin(unsigned char* smem, int warps, int warp, const CopySource* s, const RingArgs& a, int x,
		int y, int z, int z_end)
	{
		const int lane = threadIdx.x & 31;
		ring = smem + warp * (kRingStages * PLANE);
		columns = reinterpret_cast<int*>(smem + warps * (kRingStages * PLANE)) + warp * 32 * COPIES;
		y0 = y;
		z1 = z_end;
		slot = 0;
		from = 0;
		rows_in = 0;
		for (int r = 0; r < S::ROWS; ++r) {
			int yi = 0;
			const int at = y0 - R + r;
			// rows and columns that no stored output reads stay out; the others are among the plane's rows
			const bool there = at < a.ny + R && map_coord(at, a.ny, a.border, yi);
			const int to = yi - (y0 - R);
			const bool use = there && to >= 0 && to < S::ROWS;
			from |= static_cast<unsigned long long>(use ? to : 15) << (4 * r);
			if (use) rows_in |= 1u << r;
		}
		for (int k = lane; k < 32 * COPIES; k += 32) {
			int xi = 0;
			const int c = x - kRingOut + k;
			columns[k] = c < a.nx + R && map_coord(c, a.nx, a.border, xi) ? xi : -1;
		}
		__syncwarp();
		for (int k = 0; k < kRingStages - 1; ++k) copy(s, a, z + k, k);
		prepare(a);
	}

	// The copy of plane z, if there is one, into slot `to`.
	__device__ __forceinline__ void copy(const CopySource* s, const RingArgs& a, int z, int to)
	{
		const int lane = threadIdx.x & 31;
		if (z < z1) {
			int zi = 0;
			const bool inside = map_coord(z, a.nz, a.border, zi);
			const char* plane = s->src + zi * s->s_plane;
			long long at[COPIES];
			int bytes[COPIES];
#pragma unroll
			for (int k = 0; k < COPIES; ++k) {
				const int xi = columns[32 * k + lane];
				at[k] = 4LL * max(xi, 0);
				bytes[k] = inside && xi >= 0 ? 4 : 0;
			}
			float* cells = reinterpret_cast<float*>(ring + to * PLANE) + lane;
#pragma unroll 2
			for (int r = 0; r < S::ROWS; ++r, cells += 4 * S::GROUPS) {
				const int f = static_cast<int>(from >> (4 * r) & 15u);
				const bool there = SPARE ? f < S::ROWS : rows_in >> r & 1u;
				const char* row = plane + (there ? y0 - R + f : 0) * s->s_row;
#pragma unroll
				for (int k = 0; k < COPIES; ++k) {
					if (32 * k + lane < 4 * S::GROUPS) cp_async4(cells + 32 * k, row + at[k], there ? bytes[k] : 0);
				}
			}
		}
		cp_async_commit(); // empty past the end, so that prepare() can count
	}

	__device__ __forceinline__ const float4* plane(const CopySource* s, const RingArgs& a, int z)
	{
		__syncwarp();
		copy(s, a, z + kRingStages - 1, slot == 0 ? kRingStages - 1 : slot - 1);
		const float4* rows = reinterpret_cast<const float4*>(ring + slot * PLANE);
		if (++slot == kRingStages) slot = 0;
		return rows;
	}

	// plane() brings the warp together.
	__device__ __forceinline__ void prepare(const RingArgs&) { cp_async_wait<kRingStages - 2>(); }

	template<bool EDGE> __device__ __forceinline__ void read(const float4* rows, int r, float (&w)[kRingOut + 2 * R]) const
	{
		ring_row<R>(rows + r * S::GROUPS + S::own(), w);
	}
};

// Whether CopyRing can load from the view: f32 contiguous along x, 16 or more along x and y.
inline bool ring_rows(const DevView& s)
{
	return s.dtype == IANE_GB_F32 && s.stride[0] == 4 && s.ext[0] >= 16 && s.ext[1] >= 16;
}

// and WarpRing: TMA-addressable
inline bool ring_supported(const DevView& s)
{
	return ring_rows(s) && rows_aligned16(s) && s.stride[1] >= 4LL * s.ext[0] &&
		(s.ext[2] <= 1 || s.stride[2] >= s.stride[1] * s.ext[1]);
}

template<int R, int LANES> int ring_map(CUtensorMap* map, const DevView& s)
{
	return encode_tensor_map_f32(map, s.ptr, s.ext[0], s.ext[1], s.ext[2], s.stride[1],
		s.ext[2] > 1 ? s.stride[2] : s.stride[1] * s.ext[1], 4 * RingShape<R, LANES>::GROUPS, RingShape<R, LANES>::ROWS);
}

// Warps of a block, one above the other: `most`, or as many as the rows need. The kernels of 32 lanes side
// by side are compiled for `most`.
template<class Shape> int ring_warps(const RingArgs& a, int most)
{
	return Shape::LANES == 32 ? most : min(most, (a.ny + Shape::OUT_ROWS - 1) / Shape::OUT_ROWS);
}

// Blocks of `warps` warps that cover the rows and columns.
template<class Shape> dim3 ring_tiles(const RingArgs& a, int warps)
{
	return dim3((a.nx + Shape::COLUMNS - 1) / Shape::COLUMNS, (a.ny + Shape::OUT_ROWS * warps - 1) / (Shape::OUT_ROWS * warps));
}

}  // namespace iane_gb
