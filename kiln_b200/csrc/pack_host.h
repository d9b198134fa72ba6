// The vectorised inner work of the host packer (pack_host.cpp).
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace kiln {

constexpr int kHostBlockCols = 256;  // most columns of a block

bool pack_host_vectorised();  // whether this CPU has the instructions

// Quantises and packs one scale group's rows of a block of columns.  scale_row: the group's row of scales; scale_pos[c]: position
// of column c of a 64-column run within the run.
void pack_host_block(const float *weight, int n, int row0, int rows, int col0, int cols, int32_t *b_packed, uint16_t *scale_row,
                     const int *scale_pos, float *dequant);

}  // namespace kiln
