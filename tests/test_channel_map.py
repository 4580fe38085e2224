"""The tensor map that delivers Gate/Up weight rows by channel: which row lands where, for both layouts.
Host code, run by a small program against an encoder of its own."""

import os
import subprocess

import pytest

from grain_gemm_b200 import build

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "tensor_map.cuh"

static unsigned long long dims[5], strides[4], box[5];
static CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t rank, void*, const cuuint64_t* d,
                       const cuuint64_t* s, const cuuint32_t* b, const cuuint32_t*, CUtensorMapInterleave,
                       CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  for (unsigned i = 0; i < rank; ++i) dims[i] = d[i], box[i] = b[i];
  for (unsigned i = 0; i + 1 < rank; ++i) strides[i] = s[i];
  return rank == 5 ? CUDA_SUCCESS : CUDA_ERROR_INVALID_VALUE;
}

int main() {
  const int experts = 3, inter = 512, hidden = 768;
  char memory[1];
  CUtensorMap map;
  for (int interleaved = 0; interleaved < 2; ++interleaved) {
    if (gg::gate_up_channel_map(encode, &map, memory, experts, inter, hidden, interleaved)) return 1;
    // Coordinates of the kernel for expert 2, channel 128, and of the last box of the weight.
    for (int channel : {128, 384}) {
      const unsigned long long c = (interleaved ? 2 * inter + channel : 2 * 2 * inter + channel) / 16;
      std::printf("%d %d:", interleaved, channel);
      for (unsigned long long q = 0; q < box[4]; ++q)
        for (unsigned long long u = 0; u < box[3]; ++u)
          for (unsigned long long j = 0; j < box[2]; ++j)
            for (unsigned long long r = 0; r < box[1]; ++r)
              std::printf(" %llu", (r * strides[0] + j * strides[1] + u * strides[2] + (c + q) * strides[3]) / hidden);
      std::printf(" | %d\n", c + box[4] <= dims[4]);
    }
    const unsigned long long last = (dims[1] - 1) * strides[0] + (dims[2] - 1) * strides[1] +
                                    (dims[3] - 1) * strides[2] + (dims[4] - 1) * strides[3];
    std::printf("last %d: %llu\n", interleaved, last / hidden);
  }
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    folder = tmp_path_factory.mktemp("channel_map")
    (folder / "program.cpp").write_text(PROGRAM)
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.find_nvcc()))), "include")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-x", "c++", f"-I{build.CSRC}", f"-I{include}",
                    "-o", str(folder / "program"), str(folder / "program.cpp")], check=True)
    output = subprocess.run([str(folder / "program")], check=True, capture_output=True, text=True).stdout
    return dict(line.split(":", 1) for line in output.splitlines())


@pytest.mark.parametrize("channel", [128, 384])
@pytest.mark.parametrize("interleaved", [0, 1])
def test_rows_by_channel(lines, interleaved, channel):
    rows, inside = lines[f"{interleaved} {channel}"].split("|")
    expected = []
    for lane in range(256):
        quarter, up, j, r = lane // 32, lane // 16 % 2, lane // 8 % 2, lane % 8
        c = channel + 16 * quarter + 2 * r + j
        expected.append(2 * 2 * 512 + (2 * c + up if interleaved else up * 512 + c))
    assert [int(v) for v in rows.split()] == expected
    assert inside.strip() == "1"


def test_the_map_ends_with_the_weight(lines):
    assert int(lines["last 0"]) <= 3 * 2 * 512 - 1 and int(lines["last 1"]) <= 3 * 2 * 512 - 1
