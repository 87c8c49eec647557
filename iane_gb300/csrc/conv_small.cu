// FP32 convolution of small single-plane jobs: too few 64x64 tiles for the register-tiled kernel
// to fill the GPU, so what counts is the chain launch, load, sums, store.
//
// A block of 256 threads stages a 32x16 tile with its halo in shared memory as floats (any source
// type or texture, the border rule applied while loading, all of a thread's loads in flight
// together) beside the kernel's taps. A thread sums two outputs, one above the other: an input
// row is read once for both, taps come four at a time as broadcasts, and the row's products are
// unrolled for the kernel's width. The generic kernel, which took these jobs, computes an output
// per thread with two shared loads per product and runtime loops: 512x512 f32 7x7 9.8 us there,
// 5.8 here (of which launch and loads are most: the products take 0.4); 901x700 u8 7x7 20.4 and
// 10.5; 640x384 11x11 14.2 and 8.7.
//
// Taps are added in the generic kernel's order -- kernel raster order, FP32 fma from +0, every
// border sample taking part -- so the results are its bits.
#include "common.cuh"
#include "kernels.h"

namespace iane_gb {
namespace {

constexpr int SX = 32, SY = 16; // outputs of a block
constexpr int WARPS = 8;

struct SmallArgs {
	DevView src, dst;
	const char* kernel;
	long long k_stride[2];
	int ky;
	int border;
	int use_tex;
	TexSource tex;
};

template<int KX>
__global__ void __launch_bounds__(32 * WARPS) conv_small_kernel(const SmallArgs a)
{
	extern __shared__ __align__(16) float shared[];
	constexpr int RX = KX / 2, KXP = (KX + 3) & ~3;
	constexpr int TW = SX + 2 * RX;
	constexpr int COLS = (TW + 31) / 32; // columns of a row per lane
	const int ky = a.ky, ry = ky / 2;
	const int th = SY + 2 * ry;
	float* taps = shared;             // [ky][KXP], zero-padded
	float* tile = shared + ky * KXP;  // [th][TW]
	const int lane = threadIdx.x, warp = threadIdx.y, tid = warp * 32 + lane;
	const int nx = a.src.ext[0], ny = a.src.ext[1];
	const int x0 = blockIdx.x * SX, y0 = blockIdx.y * SY, z = blockIdx.z;

	// the lane's columns: element offsets, mapped once
	int xi[COLS];
	unsigned have = 0;
#pragma unroll
	for (int k = 0; k < COLS; ++k) {
		xi[k] = 0;
		if (map_coord(x0 - RX + lane + 32 * k, nx, a.border, xi[k])) have |= 1u << k;
	}
	const char* plane = a.src.ptr + z * a.src.stride[2];
#pragma unroll 3
	for (int r = warp; r < th; r += WARPS) {
		int yi = 0;
		const bool row = map_coord(y0 - ry + r, ny, a.border, yi);
		float v[COLS];
#pragma unroll
		for (int k = 0; k < COLS; ++k) {
			if (a.use_tex) {
				v[k] = texel_as_float(a.tex.tex, a.tex.dtype, a.tex.rank, a.tex.origin[0] + xi[k], a.tex.origin[1] + yi,
					a.tex.origin[2] + z);
			} else {
				v[k] = load_as_float(plane + yi * a.src.stride[1] + xi[k] * a.src.stride[0], a.src.dtype);
			}
		}
#pragma unroll
		for (int k = 0; k < COLS; ++k) {
			const int c = lane + 32 * k;
			if (c < TW) tile[r * TW + c] = row && (have >> k & 1u) ? v[k] : 0.0f;
		}
	}
	for (int i = tid; i < ky * KXP; i += 32 * WARPS) {
		const int qx = i % KXP, qy = i / KXP;
		taps[i] = qx < KX ? *reinterpret_cast<const float*>(a.kernel + qx * a.k_stride[0] + qy * a.k_stride[1]) : 0.0f;
	}
	__syncthreads();

	// outputs (x0 + lane, y0 + 2 warp) and the one below; kernel row b of output j meets tile row
	// 2 warp + j + 2 ry - b: tile rows from the last to the first give each its rows in order
	float s0 = 0.0f, s1 = 0.0f;
	const float* in = tile + (2 * warp + 1 + 2 * ry) * TW + lane;
	auto products = [&](float& s, const float (&v)[KX], int b) {
		const float4* row = reinterpret_cast<const float4*>(taps + b * KXP);
#pragma unroll
		for (int m = 0; m < KXP / 4; ++m) {
			const float4 k = row[m];
			const float kk[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				if (4 * m + i < KX) s = fmaf(v[KX - 1 - (4 * m + i)], kk[i], s);
			}
		}
	};
#pragma unroll 1
	for (int b = 0; b <= ky; ++b, in -= TW) {
		float v[KX];
#pragma unroll
		for (int i = 0; i < KX; ++i) v[i] = in[i];
		if (b < ky) products(s1, v, b);
		if (b > 0) products(s0, v, b - 1);
	}
	const int x = x0 + lane, y = y0 + 2 * warp;
	if (x >= nx) return;
	char* out = a.dst.ptr + x * a.dst.stride[0] + y * a.dst.stride[1] + z * a.dst.stride[2];
	if (y < ny) store_converted_f32(out, a.dst.dtype, s0);
	if (y + 1 < ny) store_converted_f32(out + a.dst.stride[1], a.dst.dtype, s1);
}

template<int KX>
int launch(const SmallArgs& a, cudaStream_t st)
{
	const int ry = a.ky / 2;
	const size_t smem = (static_cast<size_t>(a.ky) * ((KX + 3) & ~3) + static_cast<size_t>(SX + 2 * (KX / 2)) * (SY + 2 * ry)) * 4;
	const dim3 grid((a.src.ext[0] + SX - 1) / SX, (a.src.ext[1] + SY - 1) / SY, a.src.ext[2]);
	conv_small_kernel<KX><<<grid, dim3(32, WARPS), smem, st>>>(a); // at most 27 KB
	IANE_GB_CUDA(cudaGetLastError(), "convolve: launch small kernel");
	return IANE_GB_OK;
}

}  // namespace

int launch_conv_small(const DevView& src, const DevView& kernel, const DevView& dst, int border, cudaStream_t st,
	const TexSource* tex)
{
	if (kernel.ext[2] != 1 || kernel.ext[1] > 63) return IANE_GB_UNSUPPORTED;
	SmallArgs a{};
	a.src = src;
	a.dst = dst;
	a.kernel = kernel.ptr;
	a.k_stride[0] = kernel.stride[0];
	a.k_stride[1] = kernel.stride[1];
	a.ky = kernel.ext[1];
	a.border = border;
	if (tex) {
		a.use_tex = 1;
		a.tex = *tex;
	}
	switch (kernel.ext[0]) {
	case 1: return launch<1>(a, st);
	case 3: return launch<3>(a, st);
	case 5: return launch<5>(a, st);
	case 7: return launch<7>(a, st);
	case 9: return launch<9>(a, st);
	case 11: return launch<11>(a, st);
	case 13: return launch<13>(a, st);
	case 15: return launch<15>(a, st);
	case 17: return launch<17>(a, st);
	case 19: return launch<19>(a, st);
	case 21: return launch<21>(a, st);
	case 23: return launch<23>(a, st);
	case 25: return launch<25>(a, st);
	case 27: return launch<27>(a, st);
	case 29: return launch<29>(a, st);
	case 31: return launch<31>(a, st);
	default: return IANE_GB_UNSUPPORTED;
	}
}

}  // namespace iane_gb
