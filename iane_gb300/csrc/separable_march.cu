// Separable FP32 convolution of 3-D f32 volumes (up to nine taps per axis): warps that march down z
// on their own, as morphology_march.cu does.
//
// What bounds it: memory (8 B per voxel) and the FMA issue next to it. A block-wide kernel that
// passes every plane through shared memory three times, with two block barriers per pair of planes,
// waits at them: issue 59%, DRAM 41% of what they can. Here a lane owns 4 columns and 4 rows: it takes
// its rows and their neighbours from the warp's ring of input planes (warp_ring.cuh, two planes ahead
// by TMA, or by 4-byte copies where TMA cannot address the rows), filters each row along x, the
// columns along y, and adds the result to the 2 R unfinished outputs of every voxel along z, all in
// registers. The y and z sums are packed two columns to an instruction, taps in pairs from shared
// memory. A warp is 128 x 4 columns and rows, or 64 x 8 (ring_narrow).
// Mirror border, that kernel -> here: 512^3 3 taps 199 -> 176 us, 5 taps 255 -> 177 (89% of the
// measured HBM rate), 7 taps 307 -> 251, 9 taps 401 -> 311; 256 x 256 x 64 7 taps 21.6 -> 18.6.
// Rows of no multiple of 16 bytes: 253 x 181 x 60 3 taps 32 -> 14.5, 7 taps 63 -> 23, 511 x 401 x 301
// 7 taps 451 -> 245.
//
// Rounding points are those of successive 1-D convolutions with an f32 intermediate; x and y sums
// run from tap 0 up, the z sums from the oldest plane to the newest.
#include "kernels.h"
#include "warp_ring.cuh"

#include <type_traits>

namespace iane_gb {
namespace {

constexpr int OUT = kRingOut;
constexpr int WARPS = 4;            // warps of a block, one above the other

struct MarchArgs {
	RingArgs in;
	char* dst;
	long long d_stride[3];    // bytes
	int zc;                   // output planes of a block
	int dst16;                // destination rows contiguous and 16-byte aligned
	const char* tap_ptr[3];   // 1-D f32 device views of the taps (null: axis beyond the rank)
	long long tap_stride[3];
	int k[3];
};

template<int R, bool EDGE, class Ring>
__device__ __forceinline__ void filter_rows(const Ring& ring, const float4* plane, const float (&tx)[2 * R + 1],
	float2 (&h)[OUT + 2 * R][OUT / 2])
{
#pragma unroll
	for (int r = 0; r < OUT + 2 * R; ++r) {
		float w[OUT + 2 * R], o[OUT];
		ring.template read<EDGE>(plane, r, w);
#pragma unroll
		for (int i = 0; i < OUT; ++i) {
			float s = 0.0f;
#pragma unroll
			for (int q = 0; q <= 2 * R; ++q) s = fmaf(tx[q], w[i + 2 * R - q], s);
			o[i] = s;
		}
#pragma unroll
		for (int p = 0; p < OUT / 2; ++p) h[r][p] = make_float2(o[2 * p], o[2 * p + 1]);
	}
}

template<int R, class Ring>
__global__ void __launch_bounds__(32 * WARPS, R >= 3 ? 2 : R == 2 ? 3 : 4)
	separable_march_kernel(const __grid_constant__ typename Ring::Source source, const MarchArgs a)
{
	constexpr int K = 2 * R + 1;
	constexpr int ROWS = OUT + 2 * R;
	constexpr int PAIRS = OUT / 2;
	extern __shared__ __align__(128) unsigned char smem[];
	__shared__ float2 taps[2][K]; // (t, t) of axes 1 and 2
	const int lane = threadIdx.x, warp = threadIdx.y, warps = Ring::LANES == 32 ? WARPS : blockDim.y;
	const int nx = a.in.nx, ny = a.in.ny;
	const int xw = blockIdx.x * Ring::COLUMNS, yw = (blockIdx.y * warps + warp) * Ring::OUT_ROWS; // the warp's first
	const int x = xw + Ring::column(), y0 = yw + Ring::row();
	const int z0 = blockIdx.z * a.zc, z1 = min(a.in.nz, z0 + a.zc);

	// taps centred and zero-padded to 2 R + 1; an axis beyond the rank is the single tap 1
	auto tap = [&](int axis, int i) -> float {
		if (!a.tap_ptr[axis]) return i == R ? 1.0f : 0.0f;
		const int q = i - (R - a.k[axis] / 2);
		return q >= 0 && q < a.k[axis] ? *reinterpret_cast<const float*>(a.tap_ptr[axis] + q * a.tap_stride[axis]) : 0.0f;
	};
	float tx[K];
#pragma unroll
	for (int i = 0; i < K; ++i) tx[i] = tap(0, i);
	const int tid = warp * 32 + lane;
	if (tid < 2 * K) {
		const float t = tap(1 + tid / K, tid % K);
		taps[tid / K][tid % K] = make_float2(t, t);
	}
	__syncthreads();
	if (yw >= ny) return;
	Ring ring;
	ring.begin(smem, warps, warp, &source, a.in, xw, yw, z0 - R, z1 + R);
	const bool whole = x + OUT <= nx;
	char* const column = a.dst + x * a.d_stride[0] + y0 * a.d_stride[1];

	// unfinished outputs: pending[k] has met its first 2 R - k planes
	float2 pending[2 * R][OUT][PAIRS];
#pragma unroll
	for (int k = 0; k < 2 * R; ++k)
#pragma unroll
		for (int j = 0; j < OUT; ++j)
#pragma unroll
			for (int p = 0; p < PAIRS; ++p) pending[k][j][p] = make_float2(0.0f, 0.0f);

	for (int z = z0 - R; z < z1 + R; ++z) {
		const float4* plane = ring.plane(&source, a.in, z);
		float2 h[ROWS][PAIRS]; // every row filtered along x
		if (ring.edge) {
			filter_rows<R, true>(ring, plane, tx, h);
		} else {
			filter_rows<R, false>(ring, plane, tx, h);
		}
		if (z + 1 < z1 + R) ring.prepare(a.in);
		float2 m[OUT][PAIRS];
#pragma unroll
		for (int j = 0; j < OUT; ++j)
#pragma unroll
			for (int p = 0; p < PAIRS; ++p) m[j][p] = make_float2(0.0f, 0.0f);
#pragma unroll
		for (int q = 0; q < K; ++q) {
			const float2 t = taps[0][q];
#pragma unroll
			for (int j = 0; j < OUT; ++j)
#pragma unroll
				for (int p = 0; p < PAIRS; ++p) m[j][p] = __ffma2_rn(h[j + 2 * R - q][p], t, m[j][p]);
		}
		// input plane z meets tap q of output z - R + q: it completes the oldest and joins the others
		const int zo = z - R;
		if (zo >= z0) {
			const float2 t = taps[1][0];
			char* out = column + zo * a.d_stride[2];
#pragma unroll
			for (int j = 0; j < OUT; ++j) {
				if (y0 + j >= ny) break;
				float2 o[PAIRS];
#pragma unroll
				for (int p = 0; p < PAIRS; ++p) o[p] = __ffma2_rn(m[j][p], t, pending[0][j][p]);
				char* row = out + j * a.d_stride[1];
				if (a.dst16 && whole) {
					*reinterpret_cast<float4*>(row) = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
				} else {
					const float v[OUT] = {o[0].x, o[0].y, o[1].x, o[1].y};
#pragma unroll
					for (int i = 0; i < OUT; ++i) {
						if (x + i < nx) *reinterpret_cast<float*>(row + i * a.d_stride[0]) = v[i];
					}
				}
			}
		}
#pragma unroll
		for (int k = 0; k < 2 * R; ++k) {
			const float2 t = taps[1][k + 1];
#pragma unroll
			for (int j = 0; j < OUT; ++j)
#pragma unroll
				for (int p = 0; p < PAIRS; ++p) {
					const float2 seen = k + 1 < 2 * R ? pending[k + 1 < 2 * R ? k + 1 : 0][j][p] : make_float2(0.0f, 0.0f);
					pending[k][j][p] = __ffma2_rn(m[j][p], t, seen);
				}
		}
	}
}

template<int R, int LANES, class Ring>
int launch_ring(const DevView& s, MarchArgs a, cudaStream_t st)
{
	const int warps = ring_warps<Ring>(a.in, WARPS);
	const size_t smem = Ring::bytes(warps);
	auto kernel = separable_march_kernel<R, Ring>;
	IANE_GB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Ring::bytes(WARPS))),
		"separable: set shared memory size"); // the most, as other threads may launch in between
	typename Ring::Source source{};
	if constexpr (std::is_same_v<Ring, WarpRing<R, LANES>>) {
		const int status = ring_map<R, LANES>(&source, s);
		if (status) return status;
	} else {
		source = CopySource{s.ptr, s.stride[1], s.stride[2]};
	}
	const dim3 tiles = ring_tiles<Ring>(a.in, warps);
	a.zc = ring_chunk(static_cast<long long>(tiles.x) * tiles.y, a.in.nz, R,
		static_cast<long long>((R >= 3 ? 2 : R == 2 ? 3 : 4) * WARPS / warps) * device_sm_count());
	kernel<<<dim3(tiles.x, tiles.y, (a.in.nz + a.zc - 1) / a.zc), dim3(32, warps), smem, st>>>(source, a);
	IANE_GB_CUDA(cudaGetLastError(), "separable: launch");
	return IANE_GB_OK;
}

template<int R, int LANES>
int launch_lanes(const DevView& s, const MarchArgs& a, cudaStream_t st)
{
	return ring_supported(s) ? launch_ring<R, LANES, WarpRing<R, LANES>>(s, a, st)
		: launch_ring<R, LANES, CopyRing<R, LANES>>(s, a, st);
}

template<int R>
int launch(const DevView& s, const MarchArgs& a, cudaStream_t st)
{
	// three taps are bound by memory, which idle lanes do not use (256 x 512 rows of 300: 57 us with 32 lanes side
	// by side, 60 with 16), and nine taps' ring of 16 rows costs 4-byte copies a tenth (rows of 701: 485, 503)
	const int most = R == 1 ? 3 : R == 4 && !ring_supported(s) ? 7 : 1 << 30;
	return ring_narrow(a.in.nx, most) ? launch_lanes<R, 16>(s, a, st) : launch_lanes<R, 32>(s, a, st);
}

}  // namespace

int launch_separable_march(const DevView& src, const DevView* taps, const DevView& dst, int border, int r, cudaStream_t st)
{
	if (!ring_rows(src) || r > 4) return IANE_GB_UNSUPPORTED;
	MarchArgs a{};
	a.in = RingArgs{src.ext[0], src.ext[1], src.ext[2], border, device_status_ptr()};
	if (!a.in.status) return IANE_GB_CUDA_ERROR;
	a.dst = dst.ptr;
	for (int i = 0; i < 3; ++i) a.d_stride[i] = dst.stride[i];
	a.dst16 = rows_aligned16(dst) ? 1 : 0;
	for (int axis = 0; axis < 3; ++axis) {
		a.tap_ptr[axis] = taps[axis].ptr;
		a.tap_stride[axis] = taps[axis].stride[0];
		a.k[axis] = taps[axis].ext[0];
	}
	switch (r) {
	case 0:
	case 1: return launch<1>(src, a, st);
	case 2: return launch<2>(src, a, st);
	case 3: return launch<3>(src, a, st);
	default: return launch<4>(src, a, st);
	}
}

}  // namespace iane_gb
