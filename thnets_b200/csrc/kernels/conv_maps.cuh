// What the tensor-core convolution launchers share: TMA descriptors (cached by what they encode) and the launch knobs.
// Defined in conv_tc.cu.
#pragma once
#include <cuda.h>
#include "thb200_kernels.h"

// a plain row-major matrix [rows][cols] with a row pitch, in boxes of 128 rows x box_cols
const CUtensorMap *thb_matrix_tmap(const void *x, long rows, int cols, int ld, int dtype, int box_cols);
// the activation operand: mode 1 plain matrix, 2 im2col, 3 im2col over rows stored with their padding
const CUtensorMap *thb_activation_tmap(const thb_conv_desc *d, const void *x, int mode);
// the packed weights in boxes of box_rows output channels x 128 or 64 bytes
const CUtensorMap *thb_weights_tmap(const thb_conv_desc *d, int box_rows, int box_bytes);
// a rank-4 im2col descriptor can describe this convolution's input
bool thb_im2col_ok(const thb_conv_desc *d);

struct ThbConvLaunch {
    int pdl, test_withhold, sms, a_tma;
    int few_tiles, few_stages; // conv_few_tc.cu: THB200_FEW_TILES (most tiles of an unsplit launch, 0: off), THB200_FEW_STAGES; -1: not set
    long long wait_limit;
};
ThbConvLaunch thb_conv_launch_knobs();
