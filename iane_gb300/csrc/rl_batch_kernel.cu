// The persistent kernel of the batched Richardson-Lucy run (rl_batch.cuh): one launch takes
// every (phase, image, tile) item of the run from the device queues, waits for the item's image
// to finish its previous phase, runs the fused tiled convolution body of the item's pass and
// PSF width, and counts the tile as done for its image.
#include "rl_batch.cuh"

namespace iane_gb {
namespace {

// Shared memory: the halo tile and taps (`stage` bytes), then this.
struct BatchShared {
	BatchImage image[2]; // the descriptor of the tile in work and of the next one
	int4 tile[2];        // phase (-1: the run is over), image, x0, y0
	int2 taps[2];        // kx, ky
	uint64_t full;       // tile, taps and descriptor have landed
	// thread 0's own: the item in hand and which of its tiles comes next
	BatchItem item;
	int phase;           // of that item; -1: nothing is left
	int next;
	int cls;             // the queue it takes items from
	unsigned int issued; // tiles handed on, the -1 included
};

// The sums of one tile for its PSF width (the epilogue is applied by the caller): the body of
// conv_tile_sums for a single kernel plane.
template<int K>
__device__ __forceinline__ void tile_sums(const float* tile, const float* taps, int ky, int t, float (&acc)[kRY][kRX])
{
	constexpr int P = TileWidth<K, 2>::P;
	const int lane = t & 31, warp = t >> 5;
	const int tx = (warp & 1) * 4 + (lane & 3), ty = (warp >> 1) * 8 + (lane >> 2);
	plane_sums<K, P, kRX, kRY>(acc, tile + kRY * ty * P + kRX * tx, taps, ky / 2, ky);
}

__device__ __forceinline__ void item_sums(const float* tile, int kx, int ky, int t, float (&acc)[kRY][kRX])
{
#define IANE_GB_BATCH_KX(K) \
	case K: tile_sums<K>(tile, tile + ((TileWidth<K, 2>::P * (kBatchTile + (ky & ~1)) + 31) & ~31), ky, t, acc); break;
	switch (kx) {
	IANE_GB_BATCH_KX(1) IANE_GB_BATCH_KX(3) IANE_GB_BATCH_KX(5) IANE_GB_BATCH_KX(7)
	IANE_GB_BATCH_KX(9) IANE_GB_BATCH_KX(11) IANE_GB_BATCH_KX(13) IANE_GB_BATCH_KX(15)
	IANE_GB_BATCH_KX(17) IANE_GB_BATCH_KX(19) IANE_GB_BATCH_KX(21) IANE_GB_BATCH_KX(23)
	IANE_GB_BATCH_KX(25) IANE_GB_BATCH_KX(27) IANE_GB_BATCH_KX(29) IANE_GB_BATCH_KX(31)
	default: break;
	}
#undef IANE_GB_BATCH_KX
}

__device__ __forceinline__ unsigned int sm_id()
{
	unsigned int id;
	asm volatile("mov.u32 %0, %%smid;" : "=r"(id));
	return id;
}

// The queue with the most work left (-1: all are empty). A CTA whose queue ran dry helps there.
__device__ __forceinline__ int fullest_queue(const BatchQueues& q, const unsigned int* heads, int phases)
{
	int best = -1;
	float most = 0.0f;
	for (int c = 0; c < q.classes; ++c) {
		const unsigned int total = static_cast<unsigned int>(q.of[c].count) * static_cast<unsigned int>(phases);
		const unsigned int taken = *reinterpret_cast<const volatile unsigned int*>(heads + c);
		if (taken >= total) continue;
		const float left = static_cast<float>(total - taken) * q.of[c].cost;
		if (best < 0 || left > most) {
			best = c;
			most = left;
		}
	}
	return best;
}

// tile_pitch(kx, 2) on the device.
__device__ __forceinline__ int batch_pitch(int kx)
{
	const int rx = kx / 2, rxa = (rx + 3) & ~3;
	const int w = 64 - kRX + ((rxa - rx + kRX + kx - 1 + 3) & ~3);
	return (w & 7) == 0 ? w + 4 : w;
}

struct FeedArgs {
	const BatchImage* images;
	const BatchItem* items;
	int phases;
	BatchSync sync;
	int* status;
	unsigned char* buffer;
	BatchShared* sh;
};

// Thread 0: take the next tile in hand (the item's next one, or a new item's first).
__device__ __forceinline__ void take_tile(const FeedArgs& a, const BatchQueues& queues)
{
	BatchShared& sh = *a.sh;
	if (sh.phase >= 0 && sh.next + 1 < sh.item.count) {
		++sh.next;
		return;
	}
	int phase = -1, cls = sh.cls;
	while (cls >= 0 && !load_volatile(a.sync.abort)) {
		const BatchClass& q = queues.of[cls];
		const unsigned int count = static_cast<unsigned int>(q.count);
		const unsigned int k = atomicAdd(a.sync.queue + cls, 1u);
		if (k < count * static_cast<unsigned int>(a.phases)) {
			phase = static_cast<int>(k / count);
			sh.item = a.items[q.first + static_cast<int>(k - static_cast<unsigned int>(phase) * count)];
			sh.next = 0;
			// the item's tensor map into the descriptor cache
			const BatchImage* im = a.images + sh.item.image;
			const CUtensorMap* map = (phase & 1) ? &im->map_ratio : &im->map_est;
			asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
			break;
		}
		cls = fullest_queue(queues, a.sync.queue, a.phases);
	}
	sh.phase = phase;
	sh.cls = cls;
}

// Completions of the image's previous phases that the tile in hand needs (four warps a tile).
__device__ __forceinline__ unsigned int tile_need(const BatchShared& sh)
{
	return batch_need(sh.phase, sh.item.image_tiles);
}

// Thread 0, the buffers being free and the image's previous phase complete: hand on the tile.
__device__ __forceinline__ void issue_tile(const FeedArgs& a)
{
	BatchShared& sh = *a.sh;
	const int slot = static_cast<int>(sh.issued++ & 1u);
	const int x0 = sh.item.x0 + sh.next * kBatchTile, y0 = sh.item.y0;
	sh.tile[slot] = make_int4(sh.phase, sh.item.image, x0, y0);
	if (sh.phase < 0) {
		mbar_arrive(&sh.full);
		return;
	}
	const int kx = sh.item.kx, ky = sh.item.ky;
	sh.taps[slot] = make_int2(kx, ky);
	const BatchImage* im = a.images + sh.item.image;
	const int pass_b = sh.phase & 1;
	const uint32_t plane = static_cast<uint32_t>(batch_pitch(kx)) * static_cast<uint32_t>(kBatchTile + 2 * (ky / 2));
	const uint32_t tap_bytes = static_cast<uint32_t>(batch_tap_pitch(kx) * ky * 4);
	fence_proxy_async_global(); // the image's previous phase, written by generic stores, before TMA
	// order earlier generic-proxy reads of the buffers before the async-proxy writes
	asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
	mbar_arrive_expect_tx(&sh.full, plane * 4 + tap_bytes + static_cast<uint32_t>(sizeof(BatchImage)));
	tma_load_3d(a.buffer, pass_b ? &im->map_ratio : &im->map_est, x0 - ((kx / 2 + 3) & ~3), y0 - ky / 2, 0, &sh.full);
	bulk_copy_shared(a.buffer + ((plane + 31) & ~31u) * 4, im->taps[pass_b], tap_bytes, &sh.full);
	bulk_copy_shared(&sh.image[slot], im, static_cast<uint32_t>(sizeof(BatchImage)), &sh.full);
}

// What bounds it: the FP32 pipe for wide PSFs, latency for narrow ones.
//
// Sixteen widths of the tile body are 419 KB of code, and with one queue for the whole batch the
// four CTAs of an SM run different widths most of the time and stall on instruction fetch. With
// a queue per width an SM's CTAs all start on the width that its id gives it (SMs are shared out
// by estimated work, neighbours together, as they share instruction caches) and change only when
// that width's queue is empty. 256 images of 64..1024 pixels a side, PSFs 3..31, 30 iterations:
// 62.4 ms with one queue, largest images first, 37.7 ms with a queue per width, 33.1 ms with the
// hand-off below (and the start values, 2 ms of it, from 32 blocks per image instead of one).
//
// The steps of the hand-off are spread over the tile before: its queue and item reads run while
// that tile is still landing, its loads (tile, taps, descriptor, all asynchronous) start as soon
// as the sums have read the buffers and land during the epilogue. A tile in hand never waits for
// its image before the tile in work is counted done, so the earliest unfinished tile can always
// proceed. Each warp counts itself done: no barrier follows the epilogue. Where a phase has few tiles
// for each CTA (batch_ahead), a CTA takes the next item only then: in its hand the item would wait for
// it, and there are idle ones.
__global__ void __launch_bounds__(128, 4) batch_persistent_kernel(const BatchImage* __restrict__ images,
	const BatchItem* __restrict__ items, const __grid_constant__ BatchQueues queues, int phases, BatchSync sync,
	int* status, unsigned int stage)
{
	extern __shared__ __align__(128) unsigned char smem_raw[];
	BatchShared* sh = reinterpret_cast<BatchShared*>(smem_raw + stage);
	const FeedArgs feed{images, items, phases, sync, status, smem_raw, sh};
	const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
	if (t == 0) {
		mbar_init(&sh->full, 1);
		fence_barrier_init();
		sh->phase = -1;
		sh->issued = 0;
		sh->cls = queues.start[sm_id() % static_cast<unsigned int>(queues.sms)];
		take_tile(feed, queues);
		if (sh->phase > 0 && !wait_counter(sync.done + sh->item.image, tile_need(*sh), sync.abort, status)) sh->phase = -1;
	}
	__syncthreads();
	if (t == 0) issue_tile(feed);
	const float* tile = reinterpret_cast<const float*>(smem_raw);
	for (unsigned int n = 0;; ++n) {
		bool held = false; // thread 0: the tile after this one is in hand
		if (t == 0 && (queues.ahead || (sh->phase >= 0 && sh->next + 1 < sh->item.count))) {
			take_tile(feed, queues);
			held = true;
		}
		const bool landed = mbar_wait_bounded(&sh->full, n & 1);
		// Thread 0 comes from the queue: apart from its warp, it would sum the tile by itself and the
		// warp's other lanes after it.
		__syncwarp();
		if (!landed) {
			report_device_status(status, IANE_GB_DEVICE_TIMEOUT);
			atomicExch(sync.abort, 1);
			return;
		}
		const int slot = n & 1;
		const int4 m = sh->tile[slot];
		const int phase = m.x;
		if (phase < 0) return;
		const int2 k = sh->taps[slot];
		const BatchImage& im = sh->image[slot];
		float acc[kRY][kRX];
#pragma unroll
		for (int j = 0; j < kRY; ++j)
#pragma unroll
			for (int i = 0; i < kRX; ++i) acc[j][i] = 0.0f;
		const int wx = m.z + 32 * (warp & 1), wy = m.w + 32 * (warp >> 1);
		// a warp whose 32 x 32 outputs all lie outside the image has nothing to sum or store
		if (wx < im.epi_a.nx && wy < im.epi_a.ny) item_sums(tile, k.x, k.y, t, acc);
		__syncthreads(); // tile and taps have been read
		bool waiting = false;
		if (t == 0) {
			waiting = !held ||
				(sh->phase > 0 && !counter_reached(load_acquire(sync.done + sh->item.image), tile_need(*sh)));
			if (!waiting) issue_tile(feed);
		}
		const int xo = wx + kRX * (lane & 3), yo = wy + kRY * (lane >> 2);
		if (phase & 1) {
			EpiUpdate epi = im.epi_b;
			epi.want_stats = 0;
			epi.write_out = phase == phases - 1 && im.write_out_final;
#pragma unroll
			for (int j = 0; j < kRY; ++j) epi.row(xo, yo + j, 0, acc[j]);
		} else {
			const EpiRatio epi = im.epi_a;
#pragma unroll
			for (int j = 0; j < kRY; ++j) epi.row(xo, yo + j, 0, acc[j]);
		}
		fence_proxy_async_global(); // this thread's epilogue stores, before other tiles' TMA reads
		__syncwarp();
		if (lane == 0) {
			__threadfence();
			atomicAdd(&sync.done[m.y], 1u);
		}
		if (waiting) {
			if (!held) take_tile(feed, queues);
			// bounded: a wait that gives up aborts the run
			if (sh->phase > 0 && !wait_counter(sync.done + sh->item.image, tile_need(*sh), sync.abort, status)) sh->phase = -1;
			issue_tile(feed);
		}
	}
}

}  // namespace

size_t batch_tile_smem(int kx, int ky)
{
	const int H = kBatchTile + 2 * (ky / 2);
	const size_t plane = (static_cast<size_t>(tile_pitch(kx, 2)) * H * 4 + 127) & ~size_t(127);
	const size_t taps = (static_cast<size_t>(ky) * batch_tap_pitch(kx) * 4 + 127) & ~size_t(127);
	return plane + taps; // 2-D images: one tile buffer and one tap buffer
}

int batch_blocks_per_sm(size_t stage)
{
	const size_t total = stage + sizeof(BatchShared);
	int per_sm = 0;
	if (cudaFuncSetAttribute(batch_persistent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
	        static_cast<int>(total)) != cudaSuccess ||
	    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_persistent_kernel, 128, total) != cudaSuccess) {
		cudaGetLastError();
		return 1;
	}
	return per_sm > 0 ? per_sm : 1;
}

int launch_batch_persistent(const BatchImage* images, const BatchItem* items, const BatchQueues& queues, int phases,
	BatchSync sync, int* status, int grid, size_t stage, cudaStream_t stream)
{
	if (queues.classes <= 0 || phases <= 0) {
		return IANE_GB_OK;
	}
	const size_t total = stage + sizeof(BatchShared);
	IANE_GB_CUDA(cudaFuncSetAttribute(batch_persistent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
		static_cast<int>(total)), "batch: set shared memory size");
	batch_persistent_kernel<<<grid, 128, total, stream>>>(images, items, queues, phases, sync, status,
		static_cast<unsigned int>(stage));
	IANE_GB_CUDA(cudaGetLastError(), "batch: launch");
	return IANE_GB_OK;
}

}  // namespace iane_gb
