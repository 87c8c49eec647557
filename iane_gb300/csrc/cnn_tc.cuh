// The tensor-core 3x3x3 convolution (cnn_tc.cu) for the other CNN kernels.
#pragma once

#include "common.cuh"

#include <cstdint>

namespace iane_gb {

// conv3 on the tensor cores, from packed (iane_gb_cnn_tc_pack) or plain [co][c0 + c1][27]
// weights. Plain weights must fit in shared memory as a whole and c0, c1 be multiples of 8 (an
// operand reads whole octets): IANE_GB_UNSUPPORTED without an error where they do not.
int launch_cnn_tc(const uint16_t* x0, int c0, const uint16_t* x1, int c1, int d, int h, int w, const uint16_t* weights,
	bool packed, const float* bias, int co, uint16_t* y16, float* y32, const float* residual, int act,
	const uint16_t* mask, cudaStream_t stream);

// The weight and bias gradient (cnn_wgrad.cu), added to dw and db. `partial` holds max_chunks x
// co x (27 (c0 + c1) + 1) floats; x0, x1 and dy are 16-byte aligned.
int launch_cnn_wgrad_tc(const uint16_t* x0, int c0, const uint16_t* x1, int c1, int d, int h, int w, const uint16_t* dy,
	int co, float* dw, float* db, float* partial, int max_chunks, cudaStream_t stream);

}  // namespace iane_gb
