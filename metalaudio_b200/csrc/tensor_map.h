// Tensor maps for the tiled copies of the TMA unit, encoded on the host.
#pragma once
#include <cuda.h>
#include <stdint.h>

namespace ma {

// Tensor map of `batch` dense [rows][row_floats] float arrays `batch_stride` floats apart, with boxes of
// box_rows x box_floats; false when the array does not qualify (alignment, stride) or the driver cannot
// encode it.
bool tile_tensor_map(const float* base, int64_t row_floats, int64_t rows, int64_t batch, int64_t batch_stride,
                     int box_floats, int box_rows, CUtensorMap* map);

}  // namespace ma
