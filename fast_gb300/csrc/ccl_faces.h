// The labelling's hand-over to the area pass, on the device.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// Per label of d_labels (fast_ccl_label_device) one byte, bit d = the label
// touches face d (Dir order); d_bits: zeroed words, one byte per label.
cudaError_t ft_label_faces(const uint32_t *d_labels, int64_t nx, int64_t ny, int64_t nz, uint32_t *d_bits,
                           cudaStream_t st);
