// Flat box erosion and dilation of 2-D planes (radii up to 4 along x and y) for 8-bit, 16-bit and
// f32 elements packed along x; the definition stands in morphology.cu.
//
// What bounds it: memory, once nothing else does. The tiled kernel spends a shared-memory load
// and a compare per sample and element on bytes. Here a thread owns 8 neighbouring elements of 8
// rows (4 of 4 for f32) and keeps everything in registers: it issues the loads of all its rows
// at once, takes the x window of each row, then the y windows.
// Integers go two to a register: bytes are widened to 16 bits (a byte permute per pair), the
// neighbour along x is a permute of two registers, and one instruction takes two minima. Every
// order of taking them gives the same integer. f32 scans in the reference's order, so
// that NaN and signed zeros come out the same bits.
//
// Rows need no alignment: a thread reads whole 32-bit words and shifts by its row's remainder.
// It does so only where these words lie inside the row; threads at the ends of a row sample
// element by element with the border rule.
//
// 2560 x 1920, erosion: u8 5 x 5 26.3 us on the tiled kernel, 6.1 here (floor 1.5); f32 29.7 and 13.5
// (floor 5.8); 4096 x 4096 u8 83 and 13.2.
#include "common.cuh"
#include "kernels.h"
#include "plane_lanes.h"

#include <limits>
#include <type_traits>

namespace iane_gb {
namespace {

constexpr int ROWS = 8;    // output rows per thread of the integer kernel

struct Plane2D {
	const char* src;
	char* dst;
	long long s_row, s_plane, d_row, d_plane;
	int nx, ny;
	int rx, ry;
	int border;
	int src16, dst16; // rows start 16-byte aligned
};

// Integers, two 16-bit lanes to a register.
template<class T, bool DILATE>
struct Pairs {
	static constexpr bool kSigned = std::is_signed_v<T>;
	static __device__ __forceinline__ uint32_t take(uint32_t a, uint32_t b)
	{
		if constexpr (kSigned) return DILATE ? __vmaxs2(a, b) : __vmins2(a, b);
		return DILATE ? __vmaxu2(a, b) : __vminu2(a, b);
	}
};

// Indices of N neighbouring samples under the border rule, always in range; bit i of the result
// is set where sample i exists (clear: it is the zero value). With these no load depends on a
// branch, and a thread's loads are all in flight together.
template<int N> __device__ __forceinline__ uint32_t map_run(int first, int n, int border, int (&at)[N])
{
	uint32_t have = 0xFFFFFFFFu;
	if (first >= 0 && first + N <= n) {
#pragma unroll
		for (int i = 0; i < N; ++i) at[i] = first + i;
	} else {
#pragma unroll
		for (int i = 0; i < N; ++i) {
			int to = 0;
			if (!map_coord(first + i, n, border, to)) have &= ~(1u << i);
			at[i] = to;
		}
	}
	return have;
}

// R: the largest radius of this instantiation (rx, ry <= R).
template<class T, bool DILATE, int R>
__global__ void __launch_bounds__(kPlaneThreads) morph_plane_int_kernel(const Plane2D a)
{
	using P = Pairs<T, DILATE>;
	constexpr int PX = 8;
	constexpr int PAD = (R + 1) & ~1;                 // elements before the first, a whole number of pairs
	constexpr int NP = (PX + 2 * PAD) / 2;            // pairs of a row
	constexpr int WORDS = (PX + 2 * PAD) * sizeof(T) / 4; // 32-bit words of a row
	const int x0 = (blockIdx.x * blockDim.x + threadIdx.x) * PX;
	const int y0 = (blockIdx.y * blockDim.y + threadIdx.y) * ROWS;
	if (x0 >= a.nx || y0 >= a.ny) return;
	const char* src = a.src + static_cast<long long>(blockIdx.z) * a.s_plane;
	// whole words around the window stay inside the row (up to 3 bytes more on either side)
	constexpr int MORE = 4 / sizeof(T);
	const bool inside = x0 - PAD - MORE >= 0 && x0 + PX + PAD + MORE <= a.nx;

	int yi[ROWS + 2 * R];
	const uint32_t rows = map_run(y0 - R, a.ny, a.border, yi);
	uint32_t raw[ROWS + 2 * R][WORDS];
	if (inside) {
		const char* first = src + (x0 - PAD) * static_cast<int>(sizeof(T));
		uint32_t v[ROWS + 2 * R][WORDS + 1];
		uint32_t shift[ROWS + 2 * R];
#pragma unroll
		for (int r = 0; r < ROWS + 2 * R; ++r) {
			const uintptr_t at = reinterpret_cast<uintptr_t>(first + yi[r] * a.s_row);
			const uint32_t* w = reinterpret_cast<const uint32_t*>(at & ~uintptr_t(3));
			shift[r] = static_cast<uint32_t>(at & 3) * 8;
#pragma unroll
			for (int k = 0; k <= WORDS; ++k) v[r][k] = w[k];
		}
#pragma unroll
		for (int r = 0; r < ROWS + 2 * R; ++r) {
#pragma unroll
			for (int k = 0; k < WORDS; ++k) {
				raw[r][k] = rows >> r & 1u ? __funnelshift_r(v[r][k], v[r][k + 1], shift[r]) : 0u;
			}
		}
	} else {
		int xi[PX + 2 * PAD];
		const uint32_t cols = map_run(x0 - PAD, a.nx, a.border, xi);
#pragma unroll
		for (int r = 0; r < ROWS + 2 * R; ++r) {
			const T* row = reinterpret_cast<const T*>(src + yi[r] * a.s_row);
			T v[PX + 2 * PAD];
#pragma unroll
			for (int i = 0; i < PX + 2 * PAD; ++i) v[i] = row[xi[i]];
#pragma unroll
			for (int k = 0; k < WORDS; ++k) raw[r][k] = 0u;
#pragma unroll
			for (int i = 0; i < PX + 2 * PAD; ++i) {
				const uint32_t u = static_cast<std::make_unsigned_t<T>>(v[i]);
				if (rows >> r & cols >> i & 1u) raw[r][i * sizeof(T) / 4] |= u << (8 * (i * sizeof(T) % 4));
			}
		}
	}
	// the x window of every row
	uint32_t h[ROWS + 2 * R][PX / 2];
#pragma unroll
	for (int r = 0; r < ROWS + 2 * R; ++r) {
		uint32_t p[NP], s[NP - 1]; // pairs (2 k, 2 k + 1) and (2 k + 1, 2 k + 2)
#pragma unroll
		for (int k = 0; k < NP; ++k) {
			if constexpr (sizeof(T) == 2) {
				p[k] = raw[r][k];
			} else {
				// two bytes, zero- or sign-extended
				const uint32_t sel = P::kSigned ? (k & 1 ? 0xB3A2u : 0x9180u) : (k & 1 ? 0x4342u : 0x4140u);
				p[k] = __byte_perm(raw[r][k / 2], 0u, sel);
			}
		}
#pragma unroll
		for (int k = 0; k < NP - 1; ++k) s[k] = __byte_perm(p[k], p[k + 1], 0x5432u);
#pragma unroll
		for (int j = 0; j < PX / 2; ++j) h[r][j] = p[j + PAD / 2];
#pragma unroll
		for (int o = 1; o <= R; ++o) {
			if (o <= a.rx) {
#pragma unroll
				for (int j = 0; j < PX / 2; ++j) {
					const int lo = 2 * j + PAD - o, hi = 2 * j + PAD + o;
					h[r][j] = P::take(h[r][j], P::take(lo & 1 ? s[lo / 2] : p[lo / 2], hi & 1 ? s[hi / 2] : p[hi / 2]));
				}
			}
		}
	}
	char* dst = a.dst + static_cast<long long>(blockIdx.z) * a.d_plane;
	const bool full = x0 + PX <= a.nx;
#pragma unroll
	for (int k = 0; k < ROWS; ++k) {
		if (y0 + k >= a.ny) break;
		uint32_t m[PX / 2];
#pragma unroll
		for (int j = 0; j < PX / 2; ++j) m[j] = h[k + R][j];
#pragma unroll
		for (int o = 1; o <= R; ++o) {
			if (o <= a.ry) {
#pragma unroll
				for (int j = 0; j < PX / 2; ++j) m[j] = P::take(m[j], P::take(h[k + R - o][j], h[k + R + o][j]));
			}
		}
		T* out = reinterpret_cast<T*>(dst + (y0 + k) * a.d_row) + x0;
		const uintptr_t at = reinterpret_cast<uintptr_t>(out);
		if constexpr (sizeof(T) == 1) {
			const uint32_t w0 = __byte_perm(m[0], m[1], 0x6420u), w1 = __byte_perm(m[2], m[3], 0x6420u);
			if (full && (at & 7) == 0) {
				*reinterpret_cast<uint2*>(out) = make_uint2(w0, w1);
			} else if (full && (at & 3) == 0) {
				reinterpret_cast<uint32_t*>(out)[0] = w0;
				reinterpret_cast<uint32_t*>(out)[1] = w1;
			} else {
#pragma unroll
				for (int i = 0; i < PX; ++i) {
					if (x0 + i < a.nx) out[i] = static_cast<T>((i < 4 ? w0 : w1) >> (8 * (i & 3)));
				}
			}
		} else {
			if (full && (at & 15) == 0) {
				*reinterpret_cast<uint4*>(out) = make_uint4(m[0], m[1], m[2], m[3]);
			} else if (full && (at & 3) == 0) {
#pragma unroll
				for (int j = 0; j < PX / 2; ++j) reinterpret_cast<uint32_t*>(out)[j] = m[j];
			} else {
#pragma unroll
				for (int i = 0; i < PX; ++i) {
					if (x0 + i < a.nx) out[i] = static_cast<T>(m[i / 2] >> (16 * (i & 1)));
				}
			}
		}
	}
}

template<bool DILATE> __device__ __forceinline__ void take_f32(float v, float& r)
{
	if (DILATE ? v > r : v < r) r = v;
}

template<bool DILATE, int R>
__global__ void __launch_bounds__(kPlaneThreads) morph_plane_f32_kernel(const Plane2D a)
{
	constexpr int PX = 4, ROWS = 4;
	constexpr int N = PX + 2 * R;
	const float start = DILATE ? -std::numeric_limits<float>::infinity() : std::numeric_limits<float>::infinity();
	const int x0 = (blockIdx.x * blockDim.x + threadIdx.x) * PX;
	const int y0 = (blockIdx.y * blockDim.y + threadIdx.y) * ROWS;
	if (x0 >= a.nx || y0 >= a.ny) return;
	const char* src = a.src + static_cast<long long>(blockIdx.z) * a.s_plane;
	const bool inside = x0 - 4 >= 0 && x0 + PX + 4 <= a.nx;
	int yi[ROWS + 2 * R];
	const uint32_t rows = map_run(y0 - R, a.ny, a.border, yi);
	float v[ROWS + 2 * R][N];
	if (inside && a.src16) {
#pragma unroll
		for (int r = 0; r < ROWS + 2 * R; ++r) {
			const float4* q = reinterpret_cast<const float4*>(src + yi[r] * a.s_row) + (x0 / 4 - 1);
			const float4 q0 = q[0], q1 = q[1], q2 = q[2];
			const float w[12] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x, q2.y, q2.z, q2.w};
#pragma unroll
			for (int i = 0; i < N; ++i) v[r][i] = rows >> r & 1u ? w[4 - R + i] : 0.0f;
		}
	} else {
		int xi[N];
		const uint32_t cols = map_run(x0 - R, a.nx, a.border, xi);
#pragma unroll
		for (int r = 0; r < ROWS + 2 * R; ++r) {
			const float* row = reinterpret_cast<const float*>(src + yi[r] * a.s_row);
#pragma unroll
			for (int i = 0; i < N; ++i) v[r][i] = row[xi[i]];
		}
#pragma unroll
		for (int r = 0; r < ROWS + 2 * R; ++r) {
#pragma unroll
			for (int i = 0; i < N; ++i) v[r][i] = rows >> r & cols >> i & 1u ? v[r][i] : 0.0f;
		}
	}
	float h[ROWS + 2 * R][PX]; // the x window of every row
#pragma unroll
	for (int r = 0; r < ROWS + 2 * R; ++r) {
#pragma unroll
		for (int j = 0; j < PX; ++j) h[r][j] = start;
#pragma unroll
		for (int q = 0; q <= 2 * R; ++q) {
			const int o = DILATE ? R - q : q - R;
			if (o >= -a.rx && o <= a.rx) {
#pragma unroll
				for (int j = 0; j < PX; ++j) take_f32<DILATE>(v[r][j + R + o], h[r][j]);
			}
		}
	}
	char* dst = a.dst + static_cast<long long>(blockIdx.z) * a.d_plane;
#pragma unroll
	for (int k = 0; k < ROWS; ++k) {
		if (y0 + k >= a.ny) break;
		float m[PX];
#pragma unroll
		for (int j = 0; j < PX; ++j) m[j] = start;
#pragma unroll
		for (int q = 0; q <= 2 * R; ++q) {
			const int o = DILATE ? R - q : q - R;
			if (o >= -a.ry && o <= a.ry) {
#pragma unroll
				for (int j = 0; j < PX; ++j) take_f32<DILATE>(h[k + R + o][j], m[j]);
			}
		}
		float* out = reinterpret_cast<float*>(dst + (y0 + k) * a.d_row) + x0;
		if (a.dst16 && x0 + PX <= a.nx) {
			*reinterpret_cast<float4*>(out) = make_float4(m[0], m[1], m[2], m[3]);
		} else {
#pragma unroll
			for (int j = 0; j < PX; ++j) {
				if (x0 + j < a.nx) out[j] = m[j];
			}
		}
	}
}

bool rows16(const DevView& v)
{
	return reinterpret_cast<uintptr_t>(v.ptr) % 16 == 0 && (v.ext[1] <= 1 || v.stride[1] % 16 == 0) &&
		(v.ext[2] <= 1 || v.stride[2] % 16 == 0);
}

struct Shape {
	dim3 block, grid;
};

Shape shape_of(const Plane2D& a, int planes, bool f32, int r)
{
	const int px = f32 ? 4 : 8, rows = f32 ? 4 : ROWS;
	const int lanes = plane_lanes(a.nx, a.ny, px, rows, a.src16 != 0, r);
	const int w = lanes * px, h = kPlaneThreads / lanes * rows;
	return Shape{dim3(lanes, kPlaneThreads / lanes), dim3((a.nx + w - 1) / w, (a.ny + h - 1) / h, planes)};
}

template<class T, bool DILATE, int R>
void launch_radius(const Plane2D& a, const Shape& s, cudaStream_t st)
{
	if constexpr (std::is_same_v<T, float>) {
		morph_plane_f32_kernel<DILATE, R><<<s.grid, s.block, 0, st>>>(a);
	} else {
		morph_plane_int_kernel<T, DILATE, R><<<s.grid, s.block, 0, st>>>(a);
	}
}

template<class T, bool DILATE>
void launch_op(const Plane2D& a, const Shape& s, cudaStream_t st)
{
	const int r = a.rx > a.ry ? a.rx : a.ry;
	if (r <= 1) {
		launch_radius<T, DILATE, 1>(a, s, st);
	} else if (r == 2) {
		launch_radius<T, DILATE, 2>(a, s, st);
	} else if (r == 3) {
		launch_radius<T, DILATE, 3>(a, s, st);
	} else {
		launch_radius<T, DILATE, 4>(a, s, st);
	}
}

template<class T>
void launch_typed(const Plane2D& a, const Shape& s, bool dilate, cudaStream_t st)
{
	if (dilate) {
		launch_op<T, true>(a, s, st);
	} else {
		launch_op<T, false>(a, s, st);
	}
}

}  // namespace

int launch_morph_planes(const DevView& s, const DevView& d, const int* r, bool dilate, int border, cudaStream_t st)
{
	const int size = dtype_size(s.dtype);
	if (r[2] != 0 || r[0] > 4 || r[1] > 4 || (s.ext[0] > 1 && s.stride[0] != size) || (d.ext[0] > 1 && d.stride[0] != size)) {
		return IANE_GB_UNSUPPORTED;
	}
	Plane2D a{};
	a.src = s.ptr;
	a.dst = d.ptr;
	a.s_row = s.stride[1];
	a.s_plane = s.stride[2];
	a.d_row = d.stride[1];
	a.d_plane = d.stride[2];
	a.nx = s.ext[0];
	a.ny = s.ext[1];
	a.rx = r[0];
	a.ry = r[1];
	a.border = border;
	a.src16 = rows16(s) ? 1 : 0;
	a.dst16 = rows16(d) ? 1 : 0;
	// Radii of 3 and 4 stay on the tiled kernel where the longer threads do not pay: images too
	// small for a block per SM (300 x 256 u8, 9 x 9: 4.6 us tiled, 6.0 here; 1533 x 1001: 11.5 and
	// 7.9), and f32 rows that take a load per sample (9 x 9 on 40 planes of 513 x 300: 51 tiled, 64
	// here; 16-byte aligned rows, 2560 x 1920: 37 and 34). So do f32 windows nine wide on narrow rows or
	// less than nine tall, whose chains of compares along x the other threads of a row do not hide,
	// and windows seven wide and up to three tall on the narrowest (8e6 elements, zero border: 9 x 9 on 200
	// columns 64 us tiled, 68 here, on 512 59 and 57; 9 x 3 on 2560 42 and 47; 1 x 9 on 4000 43 and 44;
	// 7 x 1 on 60 42 and 46).
	const bool f32 = s.dtype == IANE_GB_F32;
	const int most = r[0] > r[1] ? r[0] : r[1];
	const Shape shape = shape_of(a, s.ext[2], f32, most);
	if (most > 2) {
		const long long blocks = static_cast<long long>(shape.grid.x) * shape.grid.y * shape.grid.z;
		if (blocks < device_sm_count() || (f32 && !a.src16)) return IANE_GB_UNSUPPORTED;
		if (f32 && (most == 4 ? r[0] == 0 || r[1] != 4 || a.nx < 512 : r[0] == 3 && r[1] <= 1 && a.nx < 100)) {
			return IANE_GB_UNSUPPORTED;
		}
	}
	switch (s.dtype) {
	case IANE_GB_U8: launch_typed<uint8_t>(a, shape, dilate, st); break;
	case IANE_GB_I8: launch_typed<int8_t>(a, shape, dilate, st); break;
	case IANE_GB_U16: launch_typed<uint16_t>(a, shape, dilate, st); break;
	case IANE_GB_I16: launch_typed<int16_t>(a, shape, dilate, st); break;
	case IANE_GB_F32: launch_typed<float>(a, shape, dilate, st); break;
	default: return IANE_GB_UNSUPPORTED;
	}
	IANE_GB_CUDA(cudaGetLastError(), "morphology: launch");
	return IANE_GB_OK;
}

}  // namespace iane_gb
