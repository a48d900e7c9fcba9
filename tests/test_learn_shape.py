"""Where a sample's values lie in the learner's buffers (kf_learn_shape.h, the
header the kernels index with), for batches whose buffers have more than 2^31
and 2^32 values: compiled for the host and compared with whole-number
arithmetic.  The kernels' own 32-bit thread counts stay below 2^32 for every
batch that fits 192 GB (forward) or that the bias sums' grid allows
(gradients)."""

import pathlib
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "kinectfusion_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "kf_learn_shape.h"
int main(int argc, char** argv) {
  for (int i = 1; i < argc; ++i) {
    const unsigned b = static_cast<unsigned>(std::atoll(argv[i]));
    for (const kf::Conv& c : kf::kConv) {
      std::printf("%u %zu %zu %zu\n", b, kf::input_at(c, b), kf::column_at(c, b), kf::colsum_chunks(c, b));
    }
  }
  std::printf("%d %zu\n", kf::kColsumRows, kf::kMaxColsumChunks);
}
"""

# (channels in, height, width) in, (height, width) out, im2col width
LAYERS = [((2, 60, 80), (30, 40), 24), ((32, 30, 40), (15, 20), 288), ((32, 15, 20), (8, 10), 288),
          ((64, 8, 10), (4, 5), 576)]


@pytest.fixture(scope="module")
def offsets(tmp_path_factory):
    where = tmp_path_factory.mktemp("learn_shape")
    (where / "shape.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), str(where / "shape.cpp"), "-o", str(where / "shape")],
                   check=True)

    def run(*batches):
        lines = subprocess.run([str(where / "shape"), *map(str, batches)], check=True, capture_output=True,
                               text=True).stdout.splitlines()
        return [tuple(map(int, line.split())) for line in lines]
    return run


# 24,855 and 55,925: the first samples whose column and input offsets pass 2^31
@pytest.mark.parametrize("b", [0, 8, 13_976, 24_855, 24_856, 55_924, 55_925, 99_424, 117_000])
def test_sample_offsets(offsets, b):
    *rows, _ = offsets(b)
    for row, ((cin, h, w), (oh, ow), kpad) in zip(rows, LAYERS):
        assert row == (b, b * cin * h * w, b * oh * ow * kpad, -(-b * oh * ow // 256)), row


def test_thread_counts_fit_32_bits(offsets):
    chunk_rows, max_chunks = offsets()[-1]
    assert (chunk_rows, max_chunks) == (256, 65535)  # the grid's y limit
    # forward: 1.6 MB a sample
    assert all(117_000 * (oh * ow * kpad // 8) < 2 ** 32 for _, (oh, ow), kpad in LAYERS)
    # gradients: the widest layer has 1200 rows a sample
    largest = max_chunks * chunk_rows // 1200
    assert all(largest * cin * h * w < 2 ** 32 for (cin, h, w), _, _ in LAYERS)
