// kf_learn_shape.h - the convolutions of the learned warm start and where a
// sample's values lie in their buffers.  A batch may fill the GPU's memory
// (1.6 MB a sample, over 100,000 samples in 180 GB), so a buffer has more
// values than a 32-bit index can tell apart: a sample's first value is a
// size_t, and 32 bits only count inside a sample.
#pragma once

#include <stddef.h>

#ifdef __CUDACC__
#define KF_HD __host__ __device__
#else
#define KF_HD
#endif

namespace kf {

struct Conv {
  int cin, cout, hin, win, hout, wout, k, kpad;
};
constexpr Conv kConv[4] = {{2, 32, 60, 80, 30, 40, 18, 24},
                           {32, 32, 30, 40, 15, 20, 288, 288},
                           {32, 64, 15, 20, 8, 10, 288, 288},
                           {64, 64, 8, 10, 4, 5, 576, 576}};

// Values of a sample in a layer's input (NHWC) and in its im2col matrix, and
// the first value of sample b in each.
KF_HD constexpr unsigned input_values(const Conv& c) { return static_cast<unsigned>(c.hin * c.win * c.cin); }
KF_HD constexpr unsigned column_values(const Conv& c) { return static_cast<unsigned>(c.hout * c.wout * c.kpad); }
KF_HD constexpr size_t input_at(const Conv& c, unsigned b) { return static_cast<size_t>(b) * input_values(c); }
KF_HD constexpr size_t column_at(const Conv& c, unsigned b) { return static_cast<size_t>(b) * column_values(c); }

// Rows of a bias gradient's chunk, and the chunks of a batch (the y extent of
// the gradient kernel's grid, at most 65,535).
constexpr int kColsumRows = 256;
constexpr size_t kMaxColsumChunks = 65535;
KF_HD constexpr size_t colsum_chunks(const Conv& c, unsigned batch) {
  return (static_cast<size_t>(batch) * c.hout * c.wout + kColsumRows - 1) / kColsumRows;
}

}  // namespace kf
