// Tensor-core weight gradient of the warm-start CNN's 3x3x3 convolution (tcgen05, BF16
// operands, FP32 accumulation in TMEM):
//
//     dw[co][ci][t] = sum_v dy[co](v) * x[ci](v + t - 1),     db[co] = sum_v dy[co](v)
//
// The contraction runs over voxels, K = 16 neighbours along x per MMA. In the C8 layout a voxel's
// octet of channels is 16 contiguous bytes and its right neighbour's the next 16, so rows of a
// tensor are MN-major operands as they lie: 8 voxels x 8 channels are one 128-byte core matrix,
// blocks of 8 channels follow one another at the tile's row pitch.
//
//   A (M = 128): 4 octets of x  x  4 rows y - 1 .. y + 2, one input plane, shifted along x by the
//                x tap: a descriptor start 16 bytes further, no data movement
//   B (N = 32):  2 octets of dy x  2 rows y, y + 1, one plane
//
// D[(octet, row), ch][(octet', row'), ch'] then holds tap ty = row - row' for the pairs with
// 0 <= row - row' <= 2: 6 of the 8 row pairs are wanted. The nine (tx, tz) have accumulators of
// their own, so a CTA reads each row group once for all 27 taps.
//
// The tensor cores' FP32 sums are cut off rather than rounded: the error grows with the number
// of MMAs that one accumulator takes (5.5e-9 of the result for each on random data, 6e-7 for
// the 108 of a CTA at 48 -> 16 channels and 64^3 voxels, against 2.4e-7 of FP32 arithmetic). So
// the three tz take turns in five sets of TMEM columns: after every few planes the oldest set is
// closed after at most 24 MMAs per accumulator and added to FP32 registers by the epilogue warps,
// while its tz goes on in a free set. The partials are summed in FP64: 1e-7.
//
// A CTA owns up to 32 input and 16 output channels and a share of the volume's row groups: columns of
// XK voxels x 2 rows, marched down z. An input plane and the dy plane of the same z are one
// stage; the MMAs of dy plane z need the stages of z - 1, z, z + 1. One thread loads, one issues
// MMAs, four warps sum dy for the bias gradient and empty the closed accumulator sets, combining
// the two row' of every tap (a lane shuffle), and at the end store one partial per CTA, which
// wgrad_reduce adds up in a fixed order: deterministic.
//
// What bounds it: the tensor pipe (9 MMAs of about 65 cycles per 32 voxels and 32 x 16 channels);
// measured figures stand at iane_gb_cnn_conv3_wgrad's choice of this kernel.
#include "cnn_tc.cuh"
#include "tc.cuh"

#include <algorithm>

namespace iane_gb {
namespace {

constexpr int ROWS_X = 4, ROWS_D = 2;    // rows of the operands
constexpr int OCT_X = 4, OCT_D = 2;      // and octets
constexpr int N = OCT_D * ROWS_D * 8;    // 32
constexpr int MAX_XK = 64;               // voxels of a column along x
constexpr int STAGES = 6;
constexpr int THREADS = 192;             // four warps for db and the epilogue, the loader, the MMA issuer
constexpr int COLS = 512;
constexpr int SET = 3 * N;               // columns of one tz
constexpr int SETS = 5;
constexpr int TURN = 8;                  // MMAs per accumulator between two turns; a set lives three

struct WgradTcArgs {
	int d, h, w;
	int ci, co;               // channels in all
	int groups0, groups;      // groups of OCT_X input octets, from x0 and in all
	int c0;
	int xk;                   // voxels of a column along x (a multiple of 16)
	int cols_x, cols_y;       // columns along x and y (pairs of rows)
	int zr, segments;         // dy planes of an item, items along z
	int items;                // cols_x * cols_y * segments
	int chunks;               // CTAs that share a job's items
	float* partial;           // [chunk][tz, tx][co][ty][ci], then [chunk][co] bias partials
	int* status;
};

__host__ __device__ constexpr uint32_t x_bytes(int xk) { return static_cast<uint32_t>(OCT_X * ROWS_X * (xk + 2) * 16); }
__host__ __device__ constexpr uint32_t d_bytes(int xk) { return static_cast<uint32_t>(OCT_D * ROWS_D * xk * 16); }
// the dy tile follows the x tile at a multiple of 128 bytes
__host__ __device__ constexpr uint32_t d_offset(int xk) { return (x_bytes(xk) + 127u) & ~127u; }
__host__ __device__ constexpr uint32_t stage_bytes(int xk) { return d_offset(xk) + ((d_bytes(xk) + 127u) & ~127u); }
constexpr size_t TAIL = 256 + 4 * OCT_D * 8 * sizeof(float); // barriers, TMEM address, the warps' db sums

__global__ void __launch_bounds__(THREADS) cnn_wgrad_tc_kernel(const __grid_constant__ CUtensorMap map0,
	const __grid_constant__ CUtensorMap map1, const __grid_constant__ CUtensorMap map_dy, const WgradTcArgs a)
{
	extern __shared__ __align__(128) unsigned char smem[];
	const uint32_t sb = stage_bytes(a.xk), dy_at = d_offset(a.xk);
	uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * sb);
	uint64_t* empty = full + STAGES;
	uint64_t* ready = empty + STAGES;  // [SETS] an accumulator set is closed
	uint64_t* drained = ready + SETS;  // [SETS] and has been read (four warps)
	uint32_t& tmem_base_s = *reinterpret_cast<uint32_t*>(drained + SETS);
	float* db_s = reinterpret_cast<float*>(full + 32); // [4 warps][OCT_D * 8]

	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int group = blockIdx.y, co0 = blockIdx.z * OCT_D * 8, chunk = blockIdx.x;
	const bool first_input = group < a.groups0;
	const int octet0 = (first_input ? group : group - a.groups0) * OCT_X; // within its tensor
	const bool bias = group == 0;

	if (warp == 0) tc::tmem_alloc(&tmem_base_s, COLS);
	if (tid == 32) {
		for (int s = 0; s < STAGES; ++s) {
			mbar_init(&full[s], 1);
			mbar_init(&empty[s], bias ? 5 : 1); // the MMAs, and the four warps that read dy
		}
		for (int k = 0; k < SETS; ++k) {
			mbar_init(&ready[k], 1);
			mbar_init(&drained[k], 4);
		}
		fence_barrier_init();
	}
	tc::fence_before_sync();
	__syncthreads();
	tc::fence_after_sync();
	const uint32_t tmem = tmem_base_s;
	bool ok = true;
	auto wait = [&](uint64_t* bar, uint32_t parity) {
		if (ok && !mbar_wait_bounded(bar, parity)) {
			ok = false;
			report_device_status(a.status, IANE_GB_DEVICE_TIMEOUT);
		}
	};
	// item -> origin; planes of dy z0 .. z0 + nz - 1, stages z0 - 1 .. z0 + nz
	auto origin = [&](int item, int& x0, int& y0, int& z0, int& nz) {
		const int column = item / a.segments;
		z0 = (item - column * a.segments) * a.zr;
		nz = min(a.zr, a.d - z0);
		x0 = column % a.cols_x * a.xk;
		y0 = column / a.cols_x * ROWS_D;
	};

	// dy planes of this CTA in all, and between two turns. Set number n is that of tz n % 3, in
	// columns n % SETS; turn e closes set e and opens set e + 3 (a turn with planes to come)
	int planes = 0;
	for (int item = chunk; item < a.items; item += a.chunks) {
		int x0, y0, z0, nz;
		origin(item, x0, y0, z0, nz);
		planes += nz;
	}
	const int per_turn = TURN / (a.xk / 16);

	if (warp == 4) {
		if (lane == 0) {
			const CUtensorMap* map = first_input ? &map0 : &map1;
			int slot = 0;
			uint32_t round = 0;
			for (int item = chunk; item < a.items; item += a.chunks) {
				int x0, y0, z0, nz;
				origin(item, x0, y0, z0, nz);
				for (int p = -1; p <= nz; ++p) {
					if (round > 0) wait(&empty[slot], (round - 1) & 1);
					unsigned char* st = smem + slot * sb;
					const bool has_dy = p >= 0 && p < nz;
					mbar_arrive_expect_tx(&full[slot], x_bytes(a.xk) + (has_dy ? d_bytes(a.xk) : 0u));
					// coordinates in 8-byte elements along x, two per voxel
					tma_load_4d(st, map, 2 * (x0 - 1), y0 - 1, z0 + p, octet0, &full[slot]);
					if (has_dy) tma_load_4d(st + dy_at, &map_dy, 2 * x0, y0, z0 + p, co0 / 8, &full[slot]);
					if (++slot == STAGES) {
						slot = 0;
						++round;
					}
				}
			}
		}
	} else if (warp == 5) {
		if (lane == 0) {
			// both operands MN-major (bits 15 and 16)
			const uint32_t idesc = tc::idesc_bf16_f32(128, N) | (1u << 15) | (1u << 16);
			uint32_t set[3] = {tmem, tmem + SET, tmem + 2 * SET}; // by tz
			const uint32_t x_row = static_cast<uint32_t>(a.xk + 2) * 16, d_row = static_cast<uint32_t>(a.xk) * 16;
			int slot = 0;
			uint32_t round = 0;
			bool started[3] = {false, false, false};
			int turn = 0, count = 0; // planes since the last turn
			int left = planes;
			for (int item = chunk; item < a.items; item += a.chunks) {
				int x0, y0, z0, nz;
				origin(item, x0, y0, z0, nz);
				int before = 0, centre = 0; // the two stages before this one
				for (int p = -1; p <= nz; ++p) {
					wait(&full[slot], round & 1);
					tc::fence_after_sync();
					if (p >= 1) {
						// dy plane z0 + p - 1, its input planes in `before`, `centre` and this stage
						const uint32_t base[3] = {smem_addr(smem + before * sb), smem_addr(smem + centre * sb),
							smem_addr(smem + slot * sb)};
						const uint32_t dy = base[1] + dy_at;
						for (int k = 0; k < a.xk; k += 16) {
							const uint64_t bd = tc::smem_desc(dy + static_cast<uint32_t>(k) * 16, 128, d_row);
#pragma unroll
							for (int tz = 0; tz < 3; ++tz) {
#pragma unroll
								for (int tx = 0; tx < 3; ++tx) {
									const uint64_t ad = tc::smem_desc(base[tz] + static_cast<uint32_t>(k + tx) * 16, 128, x_row);
									tc::mma_bf16(set[tz] + tx * N, ad, bd, idesc, started[tz]);
								}
								started[tz] = true;
							}
						}
						tc::commit(&empty[before]);
						--left;
						if (++count == per_turn && left > 0) {
							count = 0;
							tc::commit(&ready[turn % SETS]);
							const int next = turn + 3;
							if (next >= SETS) wait(&drained[next % SETS], (next / SETS - 1) & 1);
							tc::fence_after_sync();
#pragma unroll
							for (int tz = 0; tz < 3; ++tz) {
								if (turn % 3 == tz) {
									set[tz] = tmem + (next % SETS) * SET;
									started[tz] = false;
								}
							}
							++turn;
						}
						if (p == nz) { // the item's last stages too
							tc::commit(&empty[centre]);
							tc::commit(&empty[slot]);
						}
					}
					before = centre;
					centre = slot;
					if (++slot == STAGES) {
						slot = 0;
						++round;
					}
				}
			}
			for (int n = turn; n < turn + 3; ++n) tc::commit(&ready[n % SETS]);
		}
	} else {
		// warp = the group's octet, lane = 8 row + channel; tap ty = row sums row' = 0 here and row' = 1
		// of the row below
		float acc[3][3][OCT_D][8] = {};
		const uint32_t lanes = static_cast<uint32_t>(32 * warp) << 16;
		auto drain = [&](int n, float (&to)[3][OCT_D][8]) {
			wait(&ready[n % SETS], (n / SETS) & 1);
			__syncwarp();
			tc::fence_after_sync();
#pragma unroll
			for (int tx = 0; tx < 3; ++tx) {
#pragma unroll
				for (int o = 0; o < OCT_D; ++o) {
					float v[16];
					tc::ld_32x32b_x16(tmem + lanes + (n % SETS) * SET + tx * N + o * 16, v);
#pragma unroll
					for (int k = 0; k < 8; ++k) to[tx][o][k] += v[k] + __shfl_down_sync(0xffffffffu, v[8 + k], 8);
				}
			}
			tc::fence_before_sync();
			__syncwarp();
			if (lane == 0) mbar_arrive(&drained[n % SETS]);
		};
		auto drain_any = [&](int n) {
			if (n % 3 == 0) drain(n, acc[0]);
			else if (n % 3 == 1) drain(n, acc[1]);
			else drain(n, acc[2]);
		};
		int turn = 0, count = 0, left = planes;
		auto plane_done = [&] {
			--left;
			if (++count == per_turn && left > 0) {
				count = 0;
				drain_any(turn++);
			}
		};
		if (bias) {
			float sum[OCT_D][8] = {};
			int slot = 0;
			uint32_t round = 0;
			for (int item = chunk; item < a.items; item += a.chunks) {
				int x0, y0, z0, nz;
				origin(item, x0, y0, z0, nz);
				for (int p = -1; p <= nz; ++p) {
					wait(&full[slot], round & 1);
					if (p >= 0 && p < nz) {
						const uint4* dy = reinterpret_cast<const uint4*>(smem + slot * sb + dy_at);
#pragma unroll
						for (int o = 0; o < OCT_D; ++o) {
							for (int i = tid; i < ROWS_D * a.xk; i += 128) {
								const uint4 q = dy[o * ROWS_D * a.xk + i];
								const uint32_t v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
								for (int k = 0; k < 4; ++k) {
									sum[o][2 * k] += __uint_as_float(v[k] << 16);
									sum[o][2 * k + 1] += __uint_as_float(v[k] & 0xFFFF0000u);
								}
							}
						}
					}
					__syncwarp();
					if (lane == 0) mbar_arrive(&empty[slot]);
					if (p >= 1) plane_done(); // the MMAs of a plane come a stage after its dy
					if (++slot == STAGES) {
						slot = 0;
						++round;
					}
				}
			}
#pragma unroll
			for (int o = 0; o < OCT_D; ++o) {
#pragma unroll
				for (int k = 0; k < 8; ++k) {
					float s = sum[o][k];
					for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
					if (lane == 0) db_s[warp * OCT_D * 8 + o * 8 + k] = s;
				}
			}
			asm volatile("bar.sync 1, 128;" ::: "memory");
			if (tid < OCT_D * 8 && co0 + tid < a.co) {
				float s = 0.0f;
				for (int k = 0; k < 4; ++k) s += db_s[k * OCT_D * 8 + tid];
				a.partial[static_cast<size_t>(a.chunks) * 27 * a.co * a.ci + static_cast<size_t>(chunk) * a.co + co0 + tid] = s;
			}
		}
		if (!bias) {
			while (left > 0) plane_done();
		}
		for (int n = turn; n < turn + 3; ++n) drain_any(n);
		const int ty = lane >> 3, octet = octet0 + warp;
		const int in = (first_input ? 0 : a.c0) + octet * 8 + (lane & 7); // channel of the concatenated input
		if (ty < 3 && in < (first_input ? a.c0 : a.ci)) {
#pragma unroll
			for (int t = 0; t < 9; ++t) {
				float* out = a.partial + (((static_cast<size_t>(chunk) * 9 + t) * a.co + co0) * 3 + ty) * a.ci + in;
#pragma unroll
				for (int c = 0; c < OCT_D * 8; ++c) {
					if (co0 + c < a.co) out[static_cast<size_t>(c) * 3 * a.ci] = acc[t / 3][t % 3][c >> 3][c & 7];
				}
			}
		}
	}
	tc::fence_before_sync();
	__syncthreads();
	if (warp == 0) tc::tmem_dealloc(tmem, COLS);
}

// dw += the partials summed over the chunks in FP64, in order, four interleaved shares per element
// (threadIdx.y), and db likewise. The elements are taken in the partials' order [tz, tx][co][ty][ci].
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(const float* __restrict__ partial, int chunks, int co, int ci,
	float* dw, float* db)
{
	__shared__ double share[4][64];
	const int nw = 27 * co * ci;
	const int i = blockIdx.x * 64 + threadIdx.x;
	double s = 0.0;
	if (i < nw) {
		for (int c = threadIdx.y; c < chunks; c += 4) s += partial[static_cast<size_t>(c) * nw + i];
	} else if (i < nw + co) {
		for (int c = threadIdx.y; c < chunks; c += 4) s += partial[static_cast<size_t>(chunks) * nw + static_cast<size_t>(c) * co + (i - nw)];
	}
	share[threadIdx.y][threadIdx.x] = s;
	__syncthreads();
	if (threadIdx.y != 0 || i >= nw + co) return;
	s = (share[0][threadIdx.x] + share[1][threadIdx.x]) + (share[2][threadIdx.x] + share[3][threadIdx.x]);
	if (i >= nw) {
		if (db) db[i - nw] += static_cast<float>(s);
		return;
	}
	const int in = i % ci, ty = i / ci % 3, o = i / (3 * ci) % co, t = i / (3 * ci * co);
	dw[(static_cast<size_t>(o) * ci + in) * 27 + t % 3 + 3 * ty + 9 * (t / 3)] += static_cast<float>(s);
}

int encode_rows_map(CUtensorMap* map, const uint16_t* base, int c, int d, int h, int w, int voxels, int rows, int octets)
{
	// 8-byte elements: a row of a tile in one box line (at most 256 elements)
	const long long dims[4] = {2LL * w, h, d, (c + 7) / 8};
	const long long strides[3] = {16LL * w, 16LL * w * h, 16LL * w * h * d};
	const int box[4] = {2 * voxels, rows, 1, octets};
	return encode_tensor_map_nd(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, base, dims, strides, box);
}

}  // namespace

int launch_cnn_wgrad_tc(const uint16_t* x0, int c0, const uint16_t* x1, int c1, int d, int h, int w, const uint16_t* dy,
	int co, float* dw, float* db, float* partial, int max_chunks, cudaStream_t st)
{
	WgradTcArgs a{};
	a.status = device_status_ptr();
	if (!a.status) return IANE_GB_CUDA_ERROR;
	a.d = d;
	a.h = h;
	a.w = w;
	a.c0 = c0;
	a.ci = c0 + c1;
	a.co = co;
	a.groups0 = ((c0 + 7) / 8 + OCT_X - 1) / OCT_X;
	a.groups = a.groups0 + ((c1 + 7) / 8 + OCT_X - 1) / OCT_X;
	a.partial = partial;
	const int co_tiles = (co + OCT_D * 8 - 1) / (OCT_D * 8);
	const int jobs = a.groups * co_tiles;
	// the widest column of those that round the row up least
	int best = 0;
	for (int xk = 16; xk <= MAX_XK; xk += 16) {
		const int padded = (w + xk - 1) / xk * xk;
		if (best == 0 || padded <= best) {
			best = padded;
			a.xk = xk;
		}
	}
	a.cols_x = (w + a.xk - 1) / a.xk;
	a.cols_y = (h + ROWS_D - 1) / ROWS_D;
	const long long columns = static_cast<long long>(a.cols_x) * a.cols_y;
	if (columns * d > (1LL << 30)) return IANE_GB_UNSUPPORTED;
	// one CTA per SM over all jobs, each with a partial of its own. Items are runs of zr planes:
	// the length that ends soonest, a run costing its planes and the two more that it loads (of
	// about a quarter of the time of a plane with its MMAs)
	const long long share = std::max(1LL, std::min<long long>(max_chunks, device_sm_count() / jobs));
	double soonest = 0.0;
	for (int zr = 1; zr <= d; zr = zr < d ? std::min(2 * zr, d) : d + 1) {
		const long long items = columns * ((d + zr - 1) / zr);
		const double time = static_cast<double>((items + share - 1) / share) * (zr + 0.5);
		if (a.zr == 0 || time <= soonest) {
			soonest = time;
			a.zr = zr;
		}
	}
	a.segments = (d + a.zr - 1) / a.zr;
	a.items = static_cast<int>(columns * a.segments);
	a.chunks = static_cast<int>(std::min<long long>(share, a.items));
	CUtensorMap m0{}, m1{}, md{};
	int rc = encode_rows_map(&m0, x0, c0, d, h, w, a.xk + 2, ROWS_X, OCT_X);
	if (rc) return rc;
	rc = encode_rows_map(&m1, c1 > 0 ? x1 : x0, c1 > 0 ? c1 : c0, d, h, w, a.xk + 2, ROWS_X, OCT_X);
	if (rc) return rc;
	rc = encode_rows_map(&md, dy, co, d, h, w, a.xk, ROWS_D, OCT_D);
	if (rc) return rc;
	// a CTA takes the SM's whole TMEM: shared memory enough that no second one lands there
	auto smem_of = [](int xk) { return std::max<size_t>(STAGES * stage_bytes(xk) + TAIL, 116 * 1024); };
	const size_t smem = smem_of(a.xk);
	// the most that any width asks for, as other threads may launch between this call and the launch
	IANE_GB_CUDA(cudaFuncSetAttribute(cnn_wgrad_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
		static_cast<int>(smem_of(MAX_XK))), "cnn_conv3_wgrad: shared memory attribute");
	cnn_wgrad_tc_kernel<<<dim3(a.chunks, a.groups, co_tiles), THREADS, smem, st>>>(m0, m1, md, a);
	const int n = 27 * co * a.ci + co;
	wgrad_reduce_kernel<<<(n + 63) / 64, dim3(64, 4), 0, st>>>(partial, a.chunks, co, a.ci, dw, db);
	IANE_GB_CUDA(cudaGetLastError(), "cnn_conv3_wgrad: launch");
	return IANE_GB_OK;
}

}  // namespace iane_gb
