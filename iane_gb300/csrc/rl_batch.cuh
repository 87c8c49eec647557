// Batched Richardson-Lucy over many images of uneven size, each with its own PSF.
//
// The whole run -- every pass of every iteration of every image -- is ONE persistent launch
// over a device work queue. The queue is the list of (image, run of 64x64 tiles) items of one pass,
// repeated once per phase (phase 2t = pass A of iteration t, 2t + 1 = pass B); item k is
// (phase k / T, entry k % T) for T items per pass. CTAs (a few per SM) take items from an
// atomic counter in queue order and run the tiled FP32 convolution body with that image's TMA
// map, PSF and fused epilogue. The images of one PSF width can have a queue of their own
// (BatchClass): the CTAs of an SM then stay on one width's code until its queue is empty.
// RL's only dependency is per image: a phase of an image reads (with a halo) what the image's
// previous phase wrote and overwrites what it read, so an item of phase p waits until all
// tiles of its image's phase p - 1 are done -- a per-image completion counter that reaches
// p * 4 * tiles (modulo 2^32), counted by warps -- instead of a grid-wide drain between passes.
// Images of the next phase start as soon as their own previous pass is complete.
//
// Progress: an item waits only for items earlier in the queue, which were handed to CTAs that
// are running, so the earliest unfinished item can always proceed. Every wait is bounded (two
// seconds of global time); a wait that gives up records IANE_GB_DEVICE_TIMEOUT in the status
// word and raises an abort flag that every other wait checks, so the launch ends promptly.
//
// The CUDA graph of a run holds the counter reset, the start values and that one launch; it is
// captured on the first run and replayed while the views, scratch and parameters are unchanged.
#pragma once

#include "batch_plan.h"
#include "rl.cuh"

namespace iane_gb {

// Device-side description of one image of the batch (128-byte aligned for the maps).
struct alignas(128) BatchImage {
	CUtensorMap map_est;   // TMA map of the work estimate (pass A source)
	CUtensorMap map_ratio; // TMA map of the ratio image (pass B source)
	EpiRatio epi_a;
	EpiUpdate epi_b;       // write_out is set only in the last iteration (write_out_final)
	const float* taps[2];  // PSF and adjoint, rows padded to a multiple of four taps (16-byte aligned)
	int write_out_final;
};
static_assert(sizeof(BatchImage) % 16 == 0, "copied into shared memory in bulk");

// Device words of a run, cleared before the launch: one counter per queue, the abort flag and
// one completion counter per image.
struct BatchSync {
	unsigned int* queue;
	int* abort;
	unsigned int* done;
};

// The persistent launch (rl_batch_kernel.cu): `grid` CTAs of 128 threads, `stage` bytes of shared
// memory for a tile and its taps (batch_tile_smem over the batch).
int launch_batch_persistent(const BatchImage* images, const BatchItem* items, const BatchQueues& queues, int phases,
	BatchSync sync, int* status, int grid, size_t stage, cudaStream_t stream);

// Shared memory that a tile of PSF width kx, height ky and its taps take.
size_t batch_tile_smem(int kx, int ky);

// Resident CTAs per SM of the persistent kernel with `stage` bytes for a tile and its taps.
int batch_blocks_per_sm(size_t stage);

// Floats of one padded tap row of a PSF kx wide.
__host__ __device__ inline int batch_tap_pitch(int kx) { return (kx + 3) & ~3; }

// Fill the plan-dependent fields of one image's pass arguments and epilogues (rl.cu); the
// caller sets the buffer pointers, views and epsilon.
void rl_plan_fill_passes(const iane_gb_rl_plan* plan, TileArgs* pass_a, TileArgs* pass_b, EpiRatio* epi_a,
	EpiUpdate* epi_b, int* status);

}  // namespace iane_gb
