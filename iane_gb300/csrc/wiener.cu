// Wiener deconvolution as a prepared operation: the reference's examples/wiener/main.cu:44-83
// (2-D there; rank 1 to 3 here).
//
// prepare: the PSF is placed in an image-sized real buffer with its centre (extent / 2 per
// axis) at the origin, wrapped periodically (main.cu:112-120), transformed (FP32 real-to-
// complex; the reference's complex transform of a real image gives the same spectrum), and
// the filter G = conj(H) / (|H|^2 + noise) is formed once, in FP64 from the FP32 spectrum and
// rounded to FP32 (the reference forms the same quotient per run, main.cu:21-31).
// run: observed -> real buffer (any element type, any strides), R2C, multiply by G, C2R, and
// the result times 1 / N encoded into the destination: to_gray8 for u8
// (examples/common/deconvolution.hpp:43-55), the plain value for f32. The transforms use
// cuFFT with their work area in the caller's scratch, as the reference's FFT plans do
// (include/iane/algorithms/fft/fft.hpp:160-172); the pad, filter, multiply and encode
// kernels are this library's.
#include "common.cuh"
#include "kernels.h"

#include <cufft.h>

#include <cmath>
#include <string>

struct iane_gb_wiener_plan {
	int rank;
	int ext[3];        // image extents, axis 0 fastest (unused axes 1)
	long long n;       // real cells
	long long nc;      // complex cells of the half spectrum ((ext0 / 2 + 1) * ext1 * ext2)
	cufftHandle r2c;
	cufftHandle c2r;
	size_t work_bytes; // cuFFT work area, the larger of the two plans'
	float2* filter;    // G, nc entries
	int device;
};

namespace iane_gb {
namespace {

constexpr size_t kAlign = 256;
size_t align_up(size_t v) { return (v + kAlign - 1) & ~(kAlign - 1); }

int grid_for(long long n)
{
	const long long b = (n + 255) / 256;
	const long long cap = 16LL * device_sm_count();
	return static_cast<int>(b < 1 ? 1 : (b > cap ? cap : b));
}

// Cell p of the padded PSF: tap x with x - e/2 = p (mod n) per axis, if any.
__device__ __forceinline__ bool psf_source(int p, int n, int e, int& x)
{
	if (p < e - e / 2) {
		x = p + e / 2;
		return true;
	}
	if (p >= n - e / 2) {
		x = p - n + e / 2;
		return true;
	}
	return false;
}

__global__ void wiener_pad_psf(DevView psf, int n0, int n1, int n2, float* out)
{
	const long long total = static_cast<long long>(n0) * n1 * n2;
	for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
	     i += static_cast<long long>(gridDim.x) * blockDim.x) {
		const int p0 = static_cast<int>(i % n0);
		const int p1 = static_cast<int>((i / n0) % n1);
		const int p2 = static_cast<int>(i / (static_cast<long long>(n0) * n1));
		int x = 0, y = 0, z = 0;
		float v = 0.0f;
		if (psf_source(p0, n0, psf.ext[0], x) && psf_source(p1, n1, psf.ext[1], y) && psf_source(p2, n2, psf.ext[2], z)) {
			v = *element_ptr<float>(psf, x, y, z);
		}
		out[i] = v;
	}
}

__global__ void wiener_make_filter(float2* h, long long nc, double noise)
{
	for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < nc;
	     i += static_cast<long long>(gridDim.x) * blockDim.x) {
		const double re = h[i].x, im = h[i].y;
		const double den = re * re + im * im + noise;
		h[i] = make_float2(static_cast<float>(re / den), static_cast<float>(-im / den));
	}
}

// The copies between views and the packed transform buffer. A thread takes kGroups groups of four
// neighbouring elements of a row, all in flight together, with one load and one store per group
// where packed rows are aligned for it; blocks stride over the rows. What bounds them is memory
// (5 B per u8 pixel); with one element per thread and step they spent their time on the two
// 64-bit index divisions of each. 2560 x 1920 u8, ncu, cold: load 25 us and store 26 us then,
// 9 and 11 now. Narrow rows and small images leave most of a block without elements, and its
// latency shows: below, one element per thread (331 x 544 u8, a whole run: 29.6 us so, 31.9 by
// rows; 129 x 2600 47.6 and 52; 1200 x 700 the other way, 53 and 48).
constexpr int kGroups = 4;
constexpr int kRun = 256 * 4 * kGroups;

bool by_element(const DevView& v)
{
	const long long n = element_count(v);
	return (n < (1LL << 19) || v.ext[0] < 1024) && n < (1LL << 31);
}

// Element i of the view in packed order.
__device__ __forceinline__ char* packed_element(const DevView& v, uint32_t i)
{
	const uint32_t row = i / v.ext[0], z = row / v.ext[1];
	return v.ptr + (i - row * v.ext[0]) * v.stride[0] + (row - z * v.ext[1]) * v.stride[1] + z * v.stride[2];
}

__global__ void __launch_bounds__(256) wiener_load_element(DevView src, float* out, uint32_t n)
{
	const uint32_t i = blockIdx.x * 256u + threadIdx.x;
	if (i < n) out[i] = load_as_float(packed_element(src, i), src.dtype);
}

__global__ void __launch_bounds__(256) wiener_store_element(const float* __restrict__ real, float scale, DevView dst, uint32_t n)
{
	const uint32_t i = blockIdx.x * 256u + threadIdx.x;
	if (i < n) store_converted_f32(packed_element(dst, i), dst.dtype, real[i] * scale);
}

dim3 row_grid(const DevView& v)
{
	const long long rows = static_cast<long long>(v.ext[1]) * v.ext[2];
	return dim3((v.ext[0] + kRun - 1) / kRun, static_cast<unsigned>(rows < 65535 ? rows : 65535));
}

__global__ void __launch_bounds__(256) wiener_load(DevView src, float* out)
{
	const int nx = src.ext[0];
	const int x0 = blockIdx.x * kRun + threadIdx.x * 4;
	const bool bytes = src.dtype == IANE_GB_U8 && src.stride[0] == 1;
	const bool floats = src.dtype == IANE_GB_F32 && src.stride[0] == 4;
	for (long long row = blockIdx.y; row < static_cast<long long>(src.ext[1]) * src.ext[2]; row += gridDim.y) {
		const int z = static_cast<int>(row / src.ext[1]), y = static_cast<int>(row - static_cast<long long>(z) * src.ext[1]);
		const char* p = src.ptr + y * src.stride[1] + z * src.stride[2];
		const uintptr_t at = reinterpret_cast<uintptr_t>(p);
		const bool words = bytes && at % 4 == 0, quads = floats && at % 16 == 0;
		float v[kGroups][4];
#pragma unroll
		for (int k = 0; k < kGroups; ++k) {
			const int x = x0 + 1024 * k;
			if (words && x + 4 <= nx) {
				const uint32_t w = *reinterpret_cast<const uint32_t*>(p + x);
#pragma unroll
				for (int i = 0; i < 4; ++i) v[k][i] = static_cast<float>(w >> (8 * i) & 0xffu);
			} else if (quads && x + 4 <= nx) {
				const float4 q = *reinterpret_cast<const float4*>(p + 4LL * x);
				v[k][0] = q.x;
				v[k][1] = q.y;
				v[k][2] = q.z;
				v[k][3] = q.w;
			} else {
#pragma unroll
				for (int i = 0; i < 4; ++i) v[k][i] = x + i < nx ? load_as_float(p + (x + i) * src.stride[0], src.dtype) : 0.0f;
			}
		}
		float* o = out + row * nx;
		const bool packed = reinterpret_cast<uintptr_t>(o) % 16 == 0;
#pragma unroll
		for (int k = 0; k < kGroups; ++k) {
			const int x = x0 + 1024 * k;
			if (packed && x + 4 <= nx) {
				*reinterpret_cast<float4*>(o + x) = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
			} else {
#pragma unroll
				for (int i = 0; i < 4; ++i) {
					if (x + i < nx) o[x + i] = v[k][i];
				}
			}
		}
	}
}

__global__ void wiener_apply(float2* spec, const float2* __restrict__ g, long long nc)
{
	for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < nc;
	     i += static_cast<long long>(gridDim.x) * blockDim.x) {
		const float2 o = spec[i], w = g[i];
		spec[i] = make_float2(o.x * w.x - o.y * w.y, o.x * w.y + o.y * w.x);
	}
}

__global__ void __launch_bounds__(256) wiener_store(const float* __restrict__ real, float scale, DevView dst)
{
	const int nx = dst.ext[0];
	const int x0 = blockIdx.x * kRun + threadIdx.x * 4;
	const bool bytes = dst.dtype == IANE_GB_U8 && dst.stride[0] == 1;
	for (long long row = blockIdx.y; row < static_cast<long long>(dst.ext[1]) * dst.ext[2]; row += gridDim.y) {
		const int z = static_cast<int>(row / dst.ext[1]), y = static_cast<int>(row - static_cast<long long>(z) * dst.ext[1]);
		char* p = dst.ptr + y * dst.stride[1] + z * dst.stride[2];
		const bool words = bytes && reinterpret_cast<uintptr_t>(p) % 4 == 0;
		const float* in = real + row * nx;
		const bool packed = reinterpret_cast<uintptr_t>(in) % 16 == 0;
		float v[kGroups][4];
#pragma unroll
		for (int k = 0; k < kGroups; ++k) {
			const int x = x0 + 1024 * k;
			if (packed && x + 4 <= nx) {
				const float4 q = *reinterpret_cast<const float4*>(in + x);
				v[k][0] = q.x;
				v[k][1] = q.y;
				v[k][2] = q.z;
				v[k][3] = q.w;
			} else {
#pragma unroll
				for (int i = 0; i < 4; ++i) v[k][i] = x + i < nx ? in[x + i] : 0.0f;
			}
		}
#pragma unroll
		for (int k = 0; k < kGroups; ++k) {
			const int x = x0 + 1024 * k;
			if (words && x + 4 <= nx) {
				uint32_t w = 0;
#pragma unroll
				for (int i = 0; i < 4; ++i) w |= static_cast<uint32_t>(convert_f32_u8(v[k][i] * scale)) << (8 * i);
				*reinterpret_cast<uint32_t*>(p + x) = w;
			} else {
#pragma unroll
				for (int i = 0; i < 4; ++i) {
					if (x + i < nx) store_converted_f32(p + (x + i) * dst.stride[0], dst.dtype, v[k][i] * scale);
				}
			}
		}
	}
}

#define IANE_GB_CUFFT_OK(call, what)                                                                        \
	do {                                                                                                    \
		const cufftResult r_ = (call);                                                                      \
		if (r_ != CUFFT_SUCCESS) {                                                                          \
			return fail(IANE_GB_CUDA_ERROR, std::string(what) + ": cuFFT error " + std::to_string(static_cast<int>(r_))); \
		}                                                                                                   \
	} while (0)

int make_plans(iane_gb_wiener_plan* p)
{
	int dims[3];
	for (int i = 0; i < p->rank; ++i) dims[i] = p->ext[p->rank - 1 - i]; // slowest first
	size_t w1 = 0, w2 = 0;
	IANE_GB_CUFFT_OK(cufftCreate(&p->r2c), "wiener: FFT plan");
	IANE_GB_CUFFT_OK(cufftCreate(&p->c2r), "wiener: FFT plan");
	IANE_GB_CUFFT_OK(cufftSetAutoAllocation(p->r2c, 0), "wiener: FFT plan");
	IANE_GB_CUFFT_OK(cufftSetAutoAllocation(p->c2r, 0), "wiener: FFT plan");
	IANE_GB_CUFFT_OK(cufftMakePlanMany(p->r2c, p->rank, dims, nullptr, 1, 0, nullptr, 1, 0, CUFFT_R2C, 1, &w1),
		"wiener: FFT plan");
	IANE_GB_CUFFT_OK(cufftMakePlanMany(p->c2r, p->rank, dims, nullptr, 1, 0, nullptr, 1, 0, CUFFT_C2R, 1, &w2),
		"wiener: FFT plan");
	p->work_bytes = w1 > w2 ? w1 : w2;
	return IANE_GB_OK;
}

void destroy_plan(iane_gb_wiener_plan* p)
{
	if (!p) return;
	if (p->r2c) cufftDestroy(p->r2c);
	if (p->c2r) cufftDestroy(p->c2r);
	if (p->filter) cudaFree(p->filter);
	delete p;
}

size_t scratch_of(const iane_gb_wiener_plan* p)
{
	return align_up(static_cast<size_t>(p->n) * sizeof(float)) + align_up(static_cast<size_t>(p->nc) * sizeof(float2)) +
		align_up(p->work_bytes);
}

}  // namespace
}  // namespace iane_gb

using namespace iane_gb;

extern "C" {

int iane_gb_wiener_prepare(const iane_gb_view* psf, int rank, const int32_t* extent, float noise, void* stream,
	iane_gb_wiener_plan** plan)
{
	if (!plan || !extent) {
		return fail(IANE_GB_INVALID_ARGUMENT, "wiener prepare: null argument");
	}
	*plan = nullptr;
	// examples/wiener/main.cu:93-96, 101-104
	if (!std::isfinite(noise) || !(noise > 0.0f)) {
		return fail(IANE_GB_INVALID_ARGUMENT, "Noise must be finite and positive");
	}
	DevView k{};
	int status = normalise_view(psf, "wiener psf", &k);
	if (status) return status;
	if (k.dtype != IANE_GB_F32) {
		return fail(IANE_GB_UNSUPPORTED, "wiener prepare: the PSF is f32");
	}
	if (rank < 1 || rank > 3 || k.rank != rank) {
		return fail(IANE_GB_INVALID_ARGUMENT, "wiener prepare: the PSF needs the image's rank (1..3)");
	}
	auto* p = new iane_gb_wiener_plan{};
	p->rank = rank;
	p->n = 1;
	for (int i = 0; i < 3; ++i) {
		p->ext[i] = i < rank ? extent[i] : 1;
		if (p->ext[i] <= 0) {
			delete p;
			return fail(IANE_GB_INVALID_ARGUMENT, "wiener prepare: image extents must be positive");
		}
		if (k.ext[i] > p->ext[i] || k.ext[i] <= 0) {
			delete p;
			return fail(IANE_GB_INVALID_ARGUMENT, "PSF must fit inside the input image");
		}
		p->n *= p->ext[i];
	}
	p->nc = p->n / p->ext[0] * (p->ext[0] / 2 + 1);
	cudaGetDevice(&p->device);
	status = make_plans(p);
	if (status) {
		destroy_plan(p);
		return status;
	}
	const cudaStream_t st = static_cast<cudaStream_t>(stream);
	const cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&p->filter), static_cast<size_t>(p->nc) * sizeof(float2));
	if (e != cudaSuccess) {
		destroy_plan(p);
		return cuda_fail(e, "wiener prepare: filter");
	}
	// the PSF's spectrum, through a temporary real buffer and work area
	char* tmp = nullptr;
	const size_t real_bytes = align_up(static_cast<size_t>(p->n) * sizeof(float));
	const cudaError_t e2 = cudaMallocAsync(reinterpret_cast<void**>(&tmp), real_bytes + align_up(p->work_bytes), st);
	if (e2 != cudaSuccess) {
		destroy_plan(p);
		return cuda_fail(e2, "wiener prepare: buffers");
	}
	float* real = reinterpret_cast<float*>(tmp);
	wiener_pad_psf<<<grid_for(p->n), 256, 0, st>>>(k, p->ext[0], p->ext[1], p->ext[2], real);
	status = IANE_GB_OK;
	if (cufftSetStream(p->r2c, st) != CUFFT_SUCCESS || cufftSetWorkArea(p->r2c, tmp + real_bytes) != CUFFT_SUCCESS ||
	    cufftExecR2C(p->r2c, real, reinterpret_cast<cufftComplex*>(p->filter)) != CUFFT_SUCCESS) {
		status = fail(IANE_GB_CUDA_ERROR, "wiener prepare: PSF transform");
	}
	if (!status) {
		wiener_make_filter<<<grid_for(p->nc), 256, 0, st>>>(p->filter, p->nc, static_cast<double>(noise));
		const cudaError_t e3 = cudaGetLastError();
		if (e3 != cudaSuccess) status = cuda_fail(e3, "wiener prepare: filter kernel");
	}
	cudaFreeAsync(tmp, st);
	if (!status) {
		const cudaError_t e4 = cudaStreamSynchronize(st);
		if (e4 != cudaSuccess) status = cuda_fail(e4, "wiener prepare");
	}
	if (status) {
		destroy_plan(p);
		return status;
	}
	*plan = p;
	return IANE_GB_OK;
}

size_t iane_gb_wiener_scratch_bytes(const iane_gb_wiener_plan* plan)
{
	return plan ? scratch_of(plan) : 0;
}

int iane_gb_wiener_run(iane_gb_wiener_plan* plan, const iane_gb_view* observed, const iane_gb_view* restored,
	void* scratch, size_t scratch_bytes, void* stream)
{
	if (!plan) {
		return fail(IANE_GB_INVALID_ARGUMENT, "wiener run: null plan");
	}
	DevView s{}, d{};
	int status = normalise_view(observed, "wiener observed", &s);
	if (status) return status;
	status = normalise_view(restored, "wiener restored", &d);
	if (status) return status;
	if (s.rank != plan->rank || d.rank != plan->rank) {
		return fail(IANE_GB_INVALID_ARGUMENT, "wiener run: views need the prepared rank");
	}
	for (int i = 0; i < 3; ++i) {
		if (s.ext[i] != plan->ext[i] || d.ext[i] != plan->ext[i]) {
			return fail(IANE_GB_INVALID_ARGUMENT, "wiener run: views must match the prepared shape");
		}
	}
	if (s.dtype == IANE_GB_F64 || s.dtype == IANE_GB_RGB8 || d.dtype == IANE_GB_BF16 || d.dtype == IANE_GB_RGB8) {
		return fail(IANE_GB_UNSUPPORTED, "wiener run: observed u8/i8/u16/i16/i32/u32/bf16/f32, restored scalar");
	}
	if (!scratch || scratch_bytes < scratch_of(plan)) {
		return fail(IANE_GB_LENGTH_ERROR, "wiener run: scratch smaller than iane_gb_wiener_scratch_bytes");
	}
	const cudaStream_t st = static_cast<cudaStream_t>(stream);
	char* base = static_cast<char*>(scratch);
	float* real = reinterpret_cast<float*>(base);
	base += align_up(static_cast<size_t>(plan->n) * sizeof(float));
	cufftComplex* spec = reinterpret_cast<cufftComplex*>(base);
	base += align_up(static_cast<size_t>(plan->nc) * sizeof(float2));
	void* work = base;
	const uint32_t n = static_cast<uint32_t>(plan->n), blocks = static_cast<uint32_t>((plan->n + 255) / 256);
	if (by_element(s)) {
		wiener_load_element<<<blocks, 256, 0, st>>>(s, real, n);
	} else {
		wiener_load<<<row_grid(s), 256, 0, st>>>(s, real);
	}
	if (cufftSetStream(plan->r2c, st) != CUFFT_SUCCESS || cufftSetStream(plan->c2r, st) != CUFFT_SUCCESS ||
	    cufftSetWorkArea(plan->r2c, work) != CUFFT_SUCCESS || cufftSetWorkArea(plan->c2r, work) != CUFFT_SUCCESS ||
	    cufftExecR2C(plan->r2c, real, spec) != CUFFT_SUCCESS) {
		return fail(IANE_GB_CUDA_ERROR, "wiener run: forward transform");
	}
	wiener_apply<<<grid_for(plan->nc), 256, 0, st>>>(reinterpret_cast<float2*>(spec), plan->filter, plan->nc);
	if (cufftExecC2R(plan->c2r, spec, real) != CUFFT_SUCCESS) {
		return fail(IANE_GB_CUDA_ERROR, "wiener run: inverse transform");
	}
	// main.cu:74: scale = 1 / (w h) in double, rounded to float
	const float scale = static_cast<float>(1.0 / static_cast<double>(plan->n));
	if (by_element(d)) {
		wiener_store_element<<<blocks, 256, 0, st>>>(real, scale, d, n);
	} else {
		wiener_store<<<row_grid(d), 256, 0, st>>>(real, scale, d);
	}
	IANE_GB_CUDA(cudaGetLastError(), "wiener run: kernels");
	return IANE_GB_OK;
}

int iane_gb_wiener_destroy(iane_gb_wiener_plan* plan)
{
	destroy_plan(plan);
	return IANE_GB_OK;
}

}  // extern "C"
