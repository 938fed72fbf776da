// Between the fp32 convolutions: the one on the fp32 units (conv_f32.cu), which takes every dense layer, and the one on the tensor
// cores (conv_f32_umma.cu), which takes most of them from it.
#pragma once

#include "ops.h"

namespace pb {

// Is this layer the tensor-core kernel's?  (Its copies also want pixels and weights on 16-byte boundaries; a launch that has them elsewhere runs on the fp32
// units and reports as many blocks as were declared.)
bool conv_f32_split_layer(const pb_op_params* p);
// Modelled microseconds of a launch of up to 32 output channels on the fp32 units.
double conv_f32_units_us(const pb_op_params* p);
// Blocks and their resources (the rest of the record is the caller's).
int conv_f32_split_info(const pb_op_params* p, pb_launch_info* out);
int conv_f32_split_launch(const pb_op_params* p, const OpArgs& op, cudaStream_t st, uint32_t job_id, void* notifier, bool pdl);

// conv_umma.cu: map of the channels-last fp32 images [batch][H][W][stride], of which the first `channels` count (the others read as
// zeros), in swizzled boxes of so many channels of so many output pixels; tiled: a plain matrix of pixels (1x1 convolution).
// reach: (taps - 1) x dilation.
int encode_pixels_f32(const void* base, int channels, int stride, int W, int H, int batch, int pad_w, int pad_h, int reach_w, int reach_h, int stride_w,
                      int stride_h, bool tiled, int box_channels, int box_pixels, CUtensorMap* out);
// Map of packed fp32 weights [tap][rows][columns] in boxes of so many columns and rows of one tap.
int encode_weights_f32(const void* base, int columns, int rows, int taps, int box_columns, int box_rows, CUtensorMap* out);

}  // namespace pb
