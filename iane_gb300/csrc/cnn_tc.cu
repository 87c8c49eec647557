// Tensor-core 3x3x3 convolution of the warm-start CNN (tcgen05 implicit GEMM, BF16 operands,
// FP32 accumulation in TMEM): inference, and the training passes' convolutions with BF16 output.
//
// A tile is a block of 16 (x) x 8 (y) voxels on two z planes. For each plane the 128 voxels are
// the M rows of a GEMM with N = 16 or 32 output channels and K = input channels x taps, 16
// channels per MMA:
//
//     D_zb,tx[r, n] += sum_{ty, tz, ci} A_{ty, zb + tz}[r, ci] * W[tx, ty, tz][ci, n]
//
// where row r is the voxel (x0 - 1 + r % 16, y0 + r / 16) and A_{ty,p} the input at that voxel
// moved by ty - 1 rows in input plane p (of four). The x tap is NOT applied to the operand: each
// tx has its own accumulator and the epilogue forms out[r] = D_0[r - 1] + D_1[r] + D_2[r + 1]
// by lane shuffles, so rows r % 16 in 1..14 are outputs (14 columns per tile) and the A
// operand of every tap is the same shared-memory tile at a row offset -- a descriptor start
// address, no data movement. Every MMA reads its 4 KB A operand from shared memory, and those
// reads, not the math, bound the kernel, so all that shares an A operand is stacked along N:
// the three x taps, and for the two inner planes the two output planes they reach (input plane
// p meets tap tz = p - zb), N = 6 x (16 or 32). A K step takes 3 x 4 MMAs for its 2 x 9 taps x
// planes (13 with the first step's, which start the second plane's accumulators).
//
// Input tile: one 4-D TMA box of the C8 activation tensor, dims (x and its 8 channels, y, z,
// octet), box (128, 10, 4, 2) -> shared memory [octet][z][y][x][8 channels]: every 8
// consecutive voxels of an octet are one 128-byte K-major core matrix (LBO = the octet
// stride, SBO = 128 bytes). Out-of-range voxels and octets arrive as zeros (the padding). (With
// the channels as a dimension of their own the box is 1280 rows of 16 bytes, which the copy
// engine takes one at a time: 110 us instead of 79 for 16 -> 16 channels at 256x256x64.)
//
// Weights of a K step: [ty][8-channel half][tz = 2, 1, 0][tx][n][8], a K-major operand of 9 N
// rows per ty, of which an MMA reads 3 N or 6 N neighbouring ones. They stay in shared memory
// for all K steps where they fit (up to six steps of 32 channels): a CTA then takes many tiles
// with one copy, either packed beforehand (iane_gb_cnn_tc_pack) or gathered from the plain
// layout at its start. Otherwise each step brings its own, packed ones only.
//
// A CTA is persistent and warp specialised: one thread loads input tiles three stages ahead, one
// issues MMAs into one of two TMEM accumulator sets, four warps empty the other (bias, ReLU,
// mask, BF16 C8 store or FP32 planar store + residual). Before, each CTA took one tile with two
// stages and did load, MMAs and epilogue in turn, a plane's MMAs at a time: 16 -> 16 channels at
// 256x256x64 178 us, now 77 (268 MB there and back, 40 us); 48 -> 16 416 us, now 183; 32 -> 32
// at 128x128x32 66 us, now 38. The tensor pipe is 75% busy then: its M128 K16 MMAs take about
// 75 cycles for N = 48 and 96, more than their operand reads (44 and 56).
#include "common.cuh"
#include "cnn_tc.cuh"
#include "tc.cuh"

#include <algorithm>
#include <cstdint>

namespace iane_gb {
namespace {

constexpr int TX = 16, TY = 8;           // voxels per M tile (x, y)
constexpr int BZ = 2;                    // output planes per tile
constexpr int OUT_X = 14;                // output columns per tile
constexpr int HY = TY + 2;               // halo rows
constexpr int MAX_STAGES = 3;
constexpr int EPI_WARPS = 4;             // a quarter of the TMEM lanes each
constexpr int THREADS = 32 * (EPI_WARPS + 2); // and the loader and the MMA issuer

constexpr int A_BYTES = 2 * (BZ + 2) * HY * TX * 16;
__host__ __device__ constexpr int b_bytes(int n) { return 27 * 2 * n * 16; }
// two accumulator sets of 3 x BZ x n columns
__host__ __device__ constexpr int tmem_cols(int n) { return 2 * 3 * BZ * n <= 256 ? 256 : 512; }
constexpr size_t SMEM_MAX = 227 * 1024;
constexpr size_t TAIL_BYTES = 256; // barriers, the TMEM address and the bias

struct TcConvArgs {
	int d, h, w;
	int c0, c1;
	int steps0, steps;        // 16-channel K steps from x0, and in all
	const uint16_t* weights;  // packed: [n tile][steps][weights of a step]; plain: [co][c0 + c1][27]
	int packed;
	int resident;             // all K steps' weights stay in shared memory
	const float* bias;        // [co] or null
	int co;
	uint16_t* y16;            // C8 output or null
	float* y32;               // planar FP32 output or null
	const float* residual;    // planar FP32, added before the activation, or null
	int act;
	const uint16_t* mask;     // C8, co channels: y *= (mask > 0), or null
	int tiles_x, tiles_y, tiles; // tiles: in all
	int n_tiles;              // tiles of N output channels
	int stages;
	int* status;
};

// Element (step s, ty, half h, tz, tx, n, k) of the weights, as packed and as held in shared
// memory: w[n][ci][tx + 3 ty + 9 tz], ci the (8 h + k)-th channel of step s.
__host__ __device__ __forceinline__ int weight_at(int n_rows, int ty, int h, int tz, int tx, int n, int k)
{
	return ((((ty * 2 + h) * 3 + (2 - tz)) * 3 + tx) * n_rows + n) * 8 + k;
}

// What a launch stores: BF16, BF16 under a mask, or anything (FP32, a residual).
constexpr int kPlain = 0, kMasked = 1, kFloat = 2;

// TURNS: an accumulator takes one K step's nine MMAs and the epilogue adds the steps up in FP32
// registers. The tensor cores cut their FP32 sums off, so that the error grows with the MMAs that one
// accumulator takes; training's, whose sums were plain FP32 ones, comes no further from 64 bits this way
// (of 1.35 million BF16 results of 96 random channels, 357 are not the nearest with plain FP32 sums, 697
// with 54 MMAs in one accumulator, 175 so; of 16 channels, with nine either way, 70 and 76 of 0.68 million).
// Each set starts with one MMA more: a training layer of 48 -> 16 channels on 64^3 voxels 183.7 -> 187 us.
template<int N, int KIND, bool TURNS>
__global__ void __launch_bounds__(THREADS) cnn_tc_conv_kernel(const __grid_constant__ CUtensorMap map0,
	const __grid_constant__ CUtensorMap map1, const TcConvArgs a)
{
	extern __shared__ __align__(128) unsigned char smem[];
	constexpr uint32_t OCTET = (BZ + 2) * HY * TX * 16;  // LBO of the A operand
	constexpr uint32_t BB = b_bytes(N);
	constexpr uint32_t HALF = 9 * N * 16;                // LBO of the weights
	constexpr int COLS = tmem_cols(N);
	constexpr uint32_t SET = 3 * BZ * N;                 // columns of an accumulator set
	const int S = a.stages;
	const uint32_t stage_bytes = A_BYTES + (a.resident ? 0u : BB);
	unsigned char* const resident = smem + S * stage_bytes;
	uint64_t* bars = reinterpret_cast<uint64_t*>(resident + (a.resident ? a.steps * BB : 0u));
	uint64_t* full = bars;                 // [S] a stage has landed
	uint64_t* empty = bars + MAX_STAGES;   // [S] its MMAs are done
	uint64_t* ready = empty + MAX_STAGES;  // [2] an accumulator set is final
	uint64_t* drained = ready + 2;         // [2] and has been read (by every epilogue warp)
	uint64_t* weights_in = drained + 2;
	uint32_t& tmem_base_s = *reinterpret_cast<uint32_t*>(weights_in + 1);
	float* bias_s = reinterpret_cast<float*>(weights_in + 2); // [N], 16-byte aligned

	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int n_tile = blockIdx.x % a.n_tiles;
	const int first = blockIdx.x / a.n_tiles, stride = gridDim.x / a.n_tiles;
	const int co0 = n_tile * N;

	if (warp == 0) tc::tmem_alloc(&tmem_base_s, COLS);
	if (tid == 32) {
		for (int s = 0; s < S; ++s) {
			mbar_init(&full[s], 1);
			mbar_init(&empty[s], 1);
		}
		for (int k = 0; k < 2; ++k) {
			mbar_init(&ready[k], 1);
			mbar_init(&drained[k], EPI_WARPS);
		}
		mbar_init(weights_in, 1);
		fence_barrier_init();
	}
	if (tid >= 64 && tid < 64 + N) {
		const int c = co0 + tid - 64;
		bias_s[tid - 64] = a.bias && c < a.co ? a.bias[c] : 0.0f;
	}
	if (!a.packed) {
		// plain weights into the operand's order: rows of 16 channels x 27 taps, zero-padded
		const int ci_total = a.c0 + a.c1;
		for (int s = 0; s < a.steps; ++s) {
			uint16_t* dst = reinterpret_cast<uint16_t*>(resident + s * BB);
			const int from = s < a.steps0 ? 16 * s : a.c0 + 16 * (s - a.steps0);
			const int have = min(16, (s < a.steps0 ? a.c0 : ci_total) - from);
			for (int i = tid; i < N * 432; i += THREADS) {
				const int n = i / 432, e = i - n * 432;
				const int c = e / 27, t = e - c * 27;
				uint16_t v = 0;
				if (co0 + n < a.co && c < have) v = a.weights[(static_cast<long long>(co0 + n) * ci_total + from + c) * 27 + t];
				dst[weight_at(N, t / 3 % 3, c >> 3, t / 9, t % 3, n, c & 7)] = v;
			}
		}
		asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic stores, before the MMAs' reads
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
	auto origin = [&](int tile, int& x0, int& y0, int& z0) {
		const int row = tile / a.tiles_x;
		x0 = (tile - row * a.tiles_x) * OUT_X;
		y0 = row % a.tiles_y * TY;
		z0 = row / a.tiles_y * BZ;
	};

	if (warp == EPI_WARPS) {
		if (lane == 0) {
			const unsigned char* packed = reinterpret_cast<const unsigned char*>(a.weights) + static_cast<size_t>(n_tile) * a.steps * BB;
			if (a.packed && a.resident) {
				mbar_arrive_expect_tx(weights_in, a.steps * BB);
				for (int s = 0; s < a.steps; ++s) bulk_copy_shared(resident + s * BB, packed + static_cast<size_t>(s) * BB, BB, weights_in);
			}
			int stage = 0;
			uint32_t round = 0; // times the ring has been gone through
			for (int tile = first; tile < a.tiles; tile += stride) {
				int x0, y0, z0;
				origin(tile, x0, y0, z0);
				for (int s = 0; s < a.steps; ++s) {
					if (round > 0) wait(&empty[stage], (round - 1) & 1);
					unsigned char* st = smem + stage * stage_bytes;
					mbar_arrive_expect_tx(&full[stage], stage_bytes);
					if (s < a.steps0) {
						tma_load_4d(st, &map0, 8 * (x0 - 1), y0 - 1, z0 - 1, 2 * s, &full[stage]);
					} else {
						tma_load_4d(st, &map1, 8 * (x0 - 1), y0 - 1, z0 - 1, 2 * (s - a.steps0), &full[stage]);
					}
					if (!a.resident) bulk_copy_shared(st + A_BYTES, packed + static_cast<size_t>(s) * BB, BB, &full[stage]);
					if (++stage == S) {
						stage = 0;
						++round;
					}
				}
			}
		}
	} else if (warp == EPI_WARPS + 1) {
		if (lane == 0) {
			const uint32_t idesc3 = tc::idesc_bf16_f32(128, 3 * N), idesc6 = tc::idesc_bf16_f32(128, 6 * N);
			if (a.packed && a.resident) wait(weights_in, 0);
			int stage = 0;
			uint32_t round = 0;
			uint32_t i = 0; // sets of accumulators of this CTA so far: a tile's, or with TURNS a step's
			for (int tile = first; tile < a.tiles; tile += stride) {
				for (int s = 0; s < a.steps; ++s) {
					const bool opens = TURNS || s == 0;
					const uint32_t set = i & 1;
					if (opens && i >= 2) wait(&drained[set], (i / 2 - 1) & 1);
					wait(&full[stage], round & 1);
					tc::fence_after_sync();
					const uint32_t d0 = tmem + set * SET, d1 = d0 + 3 * N;
					const uint32_t a_base = smem_addr(smem + stage * stage_bytes);
					const uint32_t b_base = a.resident ? smem_addr(resident + s * BB) : a_base + A_BYTES;
					// input plane p reaches output plane 0 by tap tz = p and plane 1 by tz = p - 1; rows
					// of the weights from tap tz on: (2 - tz) x 3 N
#pragma unroll
					for (int p = 0; p < 4; ++p) {
#pragma unroll
						for (int ty = 0; ty < 3; ++ty) {
							const uint64_t ad = tc::smem_desc(a_base + static_cast<uint32_t>((p * HY + ty) * TX * 16), OCTET, 128);
							const uint32_t row = b_base + static_cast<uint32_t>(ty) * 2 * HALF;
							auto taps = [&](int tz) { return tc::smem_desc(row + static_cast<uint32_t>((2 - tz) * 3 * N * 16), HALF, 128); };
							if (p == 0) {
								tc::mma_bf16(d0, ad, taps(0), idesc3, !opens || ty > 0);
							} else if (p == 3) {
								tc::mma_bf16(d1, ad, taps(2), idesc3, true);
							} else if (p == 1 && ty == 0) {
								// a set's first step starts plane 1's accumulators here
								if (!opens) {
									tc::mma_bf16(d0, ad, taps(1), idesc6, true);
								} else {
									tc::mma_bf16(d0, ad, taps(1), idesc3, true);
									tc::mma_bf16(d1, ad, taps(0), idesc3, false);
								}
							} else {
								tc::mma_bf16(d0, ad, taps(p), idesc6, true);
							}
						}
					}
					tc::commit(&empty[stage]);
					if (++stage == S) {
						stage = 0;
						++round;
					}
					if (TURNS || s + 1 == a.steps) {
						tc::commit(&ready[set]);
						++i;
					}
				}
			}
			// no MMA may be in flight when the CTA gives its memory back
			if (i > 0) wait(&ready[(i - 1) & 1], ((i - 1) / 2) & 1);
		}
	} else {
		// epilogue: lane l of warp w holds row r = 32 w + l of both output planes (a second four
		// warps, one set per plane, made 16 channels slower, 79 -> 94 us at 256x256x64, and 32 no
		// faster: the tensor pipe is what is busy there)
		const int r = 32 * warp + lane;
		const long long plane = static_cast<long long>(a.h) * a.w, vol = plane * a.d;
		const uint32_t lane_base = static_cast<uint32_t>(32 * warp) << 16;
		uint32_t i = 0;
		for (int tile = first; tile < a.tiles; tile += stride) {
			int x0, y0, z0;
			origin(tile, x0, y0, z0);
			const int x = x0 - 1 + (r & 15), y = y0 + (r >> 4);
			const bool valid = (r & 15) >= 1 && (r & 15) <= OUT_X && x < a.w && y < a.h;
			const long long v0 = z0 * plane + static_cast<long long>(y) * a.w + x;
			// group q of 16 channels of a plane: the sum over the x taps
			auto group = [&](uint32_t set, int q, float (&o)[16]) {
				const int zb = q / (N / 16), j = q % (N / 16);
				__syncwarp(); // tcgen05.ld is warp-collective: lanes come from the wait or from store()
				tc::fence_after_sync();
				float d0[16], d1[16], d2[16];
				const uint32_t col = tmem + lane_base + set * SET + static_cast<uint32_t>(zb * 3 * N + 16 * j);
				tc::ld_32x32b_x16x3(col, col + N, col + 2 * N, d0, d1, d2);
				if (q == BZ * (N / 16) - 1) {
					// the set has been read: its next MMAs may have it
					tc::fence_before_sync();
					__syncwarp();
					if (lane == 0) mbar_arrive(&drained[set]);
				}
#pragma unroll
				for (int k = 0; k < 16; ++k) {
					o[k] = __shfl_up_sync(0xffffffffu, d0[k], 1) + d1[k] + __shfl_down_sync(0xffffffffu, d2[k], 1);
				}
			};
			auto store = [&](int q, float (&o)[16]) {
				const int zb = q / (N / 16), j = q % (N / 16);
				const long long v = zb ? v0 + plane : v0;
				if (!valid || z0 + zb >= a.d) return;
				const int c0 = co0 + 16 * j;
#pragma unroll
				for (int k = 0; k < 16; k += 4) {
					const float4 bias = *reinterpret_cast<const float4*>(bias_s + 16 * j + k);
					o[k] += bias.x;
					o[k + 1] += bias.y;
					o[k + 2] += bias.z;
					o[k + 3] += bias.w;
				}
				if constexpr (KIND == kFloat) {
#pragma unroll
					for (int k = 0; k < 16; ++k) {
						if (a.residual && c0 + k < a.co) o[k] += a.residual[(c0 + k) * vol + v];
					}
				}
				if (a.act == 1) {
#pragma unroll
					for (int k = 0; k < 16; ++k) o[k] = o[k] > 0.0f ? o[k] : 0.0f;
				}
				if constexpr (KIND == kFloat) {
#pragma unroll
					for (int k = 0; k < 16; ++k) {
						if (a.y32 && c0 + k < a.co) a.y32[(c0 + k) * vol + v] = o[k];
					}
				}
				if (KIND != kFloat || a.y16) {
#pragma unroll
					for (int h = 0; h < 2; ++h) {
						if (c0 + 8 * h >= a.co) break;
						const long long at = ((c0 / 8 + h) * vol + v) << 3;
						uint32_t u[4];
#pragma unroll
						for (int k = 0; k < 4; ++k) {
							const __nv_bfloat162 two = __floats2bfloat162_rn(o[8 * h + 2 * k], o[8 * h + 2 * k + 1]);
							u[k] = *reinterpret_cast<const uint32_t*>(&two);
						}
						if constexpr (KIND == kMasked) {
							// a channel's bits survive where the mask's is above zero
							const uint4 m = *reinterpret_cast<const uint4*>(a.mask + at);
							const uint32_t mw[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
							for (int k = 0; k < 4; ++k) {
								u[k] &= (__uint_as_float(mw[k] << 16) > 0.0f ? 0xFFFFu : 0u) |
									(__uint_as_float(mw[k] & 0xFFFF0000u) > 0.0f ? 0xFFFF0000u : 0u);
							}
						}
						*reinterpret_cast<uint4*>(a.y16 + at) = make_uint4(u[0], u[1], u[2], u[3]);
					}
				}
			};
			if constexpr (TURNS) {
				float sum[BZ * (N / 16)][16];
				for (int s = 0; s < a.steps; ++s, ++i) {
					wait(&ready[i & 1], (i / 2) & 1);
#pragma unroll
					for (int q = 0; q < BZ * (N / 16); ++q) {
						float o[16];
						group(i & 1, q, o);
#pragma unroll
						for (int k = 0; k < 16; ++k) sum[q][k] = s > 0 ? sum[q][k] + o[k] : o[k];
					}
				}
#pragma unroll
				for (int q = 0; q < BZ * (N / 16); ++q) store(q, sum[q]);
			} else {
				const uint32_t set = i & 1;
				wait(&ready[set], (i / 2) & 1);
#pragma unroll 1
				for (int q = 0; q < BZ * (N / 16); ++q) {
					float o[16];
					group(set, q, o);
					store(q, o);
				}
				++i;
			}
		}
	}
	tc::fence_before_sync();
	__syncthreads();
	if (warp == 0) tc::tmem_dealloc(tmem, COLS);
}

// Weights in the operand's order for every tile of n_rows output channels (weight_at).
__global__ void pack_kernel(const uint16_t* w, int co, int c0, int c1, int n_rows, int n_tiles, int steps0, int steps,
	uint16_t* packed)
{
	const int ci_total = c0 + c1;
	const long long n = static_cast<long long>(n_tiles) * steps * n_rows * 432;
	for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
	     i += static_cast<long long>(gridDim.x) * blockDim.x) {
		const int e = static_cast<int>(i % 432), row = static_cast<int>(i / 432 % n_rows);
		const long long block = i / (432LL * n_rows); // (n tile, step)
		const int s = static_cast<int>(block % steps), o = static_cast<int>(block / steps) * n_rows + row;
		const int c = e / 27, t = e - c * 27;
		const int local = 16 * (s < steps0 ? s : s - steps0) + c;
		const int ci = s < steps0 ? (local < c0 ? local : -1) : (local < c1 ? c0 + local : -1);
		packed[block * 432 * n_rows + weight_at(n_rows, t / 3 % 3, c >> 3, t / 9, t % 3, row, c & 7)] =
			(o < co && ci >= 0) ? w[(static_cast<long long>(o) * ci_total + ci) * 27 + t] : 0;
	}
}

int steps_of(int c) { return (c + 15) / 16; }

// Output channels of a tile: 16 where that is all there is (two CTAs per SM), else 32 (64
// channels of the deepest level are two tiles, which also gives its few voxels more CTAs).
int n_of(int co) { return co <= 16 ? 16 : 32; }
int n_tiles_of(int co) { return (co + n_of(co) - 1) / n_of(co); }

template<int N>
int launch(const CUtensorMap& m0, const CUtensorMap& m1, TcConvArgs a, cudaStream_t st)
{
	// plain weights are training's, whose results are BF16; packed ones inference's, without a mask
	const auto kernel = !a.packed ? a.mask ? cnn_tc_conv_kernel<N, kMasked, true> : cnn_tc_conv_kernel<N, kPlain, true>
		: a.y32 || a.residual ? cnn_tc_conv_kernel<N, kFloat, false> : cnn_tc_conv_kernel<N, kPlain, false>;
	// weights resident beside two or three input stages, or a stage of both at a time
	const size_t weights = static_cast<size_t>(a.steps) * b_bytes(N);
	// CTAs per SM are bounded by TMEM (512 columns per SM): ask for enough shared memory that
	// no more CTAs than that land on an SM (228 KB per SM, 1 KB reserved per CTA)
	const int per_sm = 512 / tmem_cols(N);
	const size_t share = SMEM_MAX / per_sm - 1024;
	const size_t most = weights + 2 * A_BYTES + TAIL_BYTES <= share ? share : SMEM_MAX;
	a.resident = weights + 2 * A_BYTES + TAIL_BYTES <= most ? 1 : 0;
	if (!a.resident && !a.packed) return IANE_GB_UNSUPPORTED;
	const size_t stage = A_BYTES + (a.resident ? 0 : b_bytes(N));
	const size_t fixed = TAIL_BYTES + (a.resident ? weights : 0);
	a.stages = static_cast<int>(std::min<size_t>(MAX_STAGES, (most - fixed) / stage));
	size_t smem = fixed + a.stages * stage;
	const size_t floor_bytes = 228 * 1024 / (per_sm + 1) - 1024 + 16;
	if (smem < floor_bytes) smem = floor_bytes;
	IANE_GB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SMEM_MAX)),
		"cnn_conv3_tc: shared memory attribute");
	// persistent: as many CTAs as are resident, the same number for each tile of channels
	const long long resident_ctas = static_cast<long long>(device_sm_count()) * (smem > share ? 1 : per_sm);
	const long long per_n = std::max(1LL, std::min<long long>(a.tiles, resident_ctas / a.n_tiles));
	kernel<<<static_cast<unsigned>(per_n * a.n_tiles), THREADS, smem, st>>>(m0, m1, a);
	IANE_GB_CUDA(cudaGetLastError(), "cnn_conv3_tc: launch");
	return IANE_GB_OK;
}

int encode_c8_map(CUtensorMap* map, const uint16_t* base, int c, int d, int h, int w)
{
	const long long dims[4] = {8LL * w, h, d, (c + 7) / 8};
	const long long strides[3] = {16LL * w, 16LL * w * h, 16LL * w * h * d};
	const int box[4] = {8 * TX, HY, BZ + 2, 2};
	return encode_tensor_map_nd(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, base, dims, strides, box);
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

}  // namespace

int launch_cnn_tc(const uint16_t* x0, int c0, const uint16_t* x1, int c1, int d, int h, int w, const uint16_t* weights,
	bool packed, const float* bias, int co, uint16_t* y16, float* y32, const float* residual, int act,
	const uint16_t* mask, cudaStream_t st)
{
	int* status = device_status_ptr();
	if (!status) return IANE_GB_CUDA_ERROR;
	TcConvArgs a{};
	a.d = d;
	a.h = h;
	a.w = w;
	a.c0 = c0;
	a.c1 = c1;
	a.steps0 = steps_of(c0);
	a.steps = a.steps0 + steps_of(c1);
	a.weights = weights;
	a.packed = packed ? 1 : 0;
	a.bias = bias;
	a.co = co;
	a.y16 = y16;
	a.y32 = y32;
	a.residual = residual;
	a.act = act;
	a.mask = mask;
	a.tiles_x = (w + OUT_X - 1) / OUT_X;
	a.tiles_y = (h + TY - 1) / TY;
	const long long tiles = static_cast<long long>(a.tiles_x) * a.tiles_y * ((d + BZ - 1) / BZ);
	if (tiles > (1LL << 30)) return IANE_GB_UNSUPPORTED;
	a.tiles = static_cast<int>(tiles);
	a.n_tiles = n_tiles_of(co);
	a.status = status;
	CUtensorMap m0{}, m1{};
	int rc = encode_c8_map(&m0, x0, c0, d, h, w);
	if (rc) return rc;
	rc = encode_c8_map(&m1, c1 > 0 ? x1 : x0, c1 > 0 ? c1 : c0, d, h, w);
	if (rc) return rc;
	return n_of(co) == 16 ? launch<16>(m0, m1, a, st) : launch<32>(m0, m1, a, st);
}

}  // namespace iane_gb

using namespace iane_gb;

extern "C" {

size_t iane_gb_cnn_tc_packed_bytes(int co, int c0, int c1)
{
	if (co < 1 || co > 64 || c0 < 1 || c1 < 0) return 0;
	return static_cast<size_t>(n_tiles_of(co)) * (steps_of(c0) + steps_of(c1)) * b_bytes(n_of(co));
}

int iane_gb_cnn_tc_pack(const uint16_t* weights, int co, int c0, int c1, uint16_t* packed, void* stream)
{
	if (!weights || !packed || co < 1 || co > 64 || c0 < 1 || c1 < 0) {
		return fail(IANE_GB_INVALID_ARGUMENT, "cnn_tc_pack: bad arguments");
	}
	const int steps0 = steps_of(c0), steps = steps0 + steps_of(c1);
	const long long n = static_cast<long long>(n_tiles_of(co)) * steps * n_of(co) * 432;
	const int grid = static_cast<int>((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
	pack_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(weights, co, c0, c1, n_of(co), n_tiles_of(co), steps0,
		steps, packed);
	IANE_GB_CUDA(cudaGetLastError(), "cnn_tc_pack: launch");
	return IANE_GB_OK;
}

int iane_gb_cnn_conv3_tc(const uint16_t* x0, int c0, const uint16_t* x1, int c1, int d, int h, int w,
	const uint16_t* packed, const float* bias, int co, uint16_t* y16, float* y32, const float* residual, int act,
	void* stream)
{
	if (!x0 || c0 < 1 || c1 < 0 || (c1 > 0 && (!x1 || c0 % 16 != 0)) || d < 1 || h < 1 || w < 1 || !packed || co < 1 ||
	    co > 64 || (!y16 && !y32) || (residual && co != 1) || (y16 && co % 8 != 0)) {
		return fail(IANE_GB_INVALID_ARGUMENT, "cnn_conv3_tc: bad arguments");
	}
	if (!aligned16(x0) || !aligned16(x1) || !aligned16(packed) || !aligned16(y16)) {
		return fail(IANE_GB_INVALID_ARGUMENT, "cnn_conv3_tc: buffers must be 16-byte aligned");
	}
	const int rc = launch_cnn_tc(x0, c0, x1, c1, d, h, w, packed, true, bias, co, y16, y32, residual, act, nullptr,
		static_cast<cudaStream_t>(stream));
	return rc == IANE_GB_UNSUPPORTED ? fail(rc, "cnn_conv3_tc: volume too large") : rc;
}

}  // extern "C"
