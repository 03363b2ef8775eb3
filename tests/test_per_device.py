"""What belongs to a device is asked of each device (``csrc/per_device.cuh``), against a stand-in for the CUDA runtime."""

import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "miniserve_b200" / "csrc"
CUDA = next((p for p in (Path("/usr/local/cuda/include"), Path(shutil.which("nvcc") or "/none").resolve().parent.parent / "include") if p.is_dir()), None)

PROGRAM = r"""
#include "per_device.cuh"
#include <cstdio>
static int device = 0, asked[100], counted[100], refuse = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int d) { ++counted[d]; *v = 100 + d; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int bytes) {
  if (refuse) return cudaErrorInvalidValue;
  asked[device] += bytes;
  return cudaSuccess;
}
int main() {
  std::atomic<unsigned long long> allowed{0};
  const int devices[] = {0, 1, 63, 64};
  refuse = 1;
  if (ms::allow_shared_memory(&device, 7, allowed) == cudaSuccess) return 1;
  refuse = 0;
  for (int round = 0; round < 3; ++round)
    for (int d : devices) {
      device = d;
      if (ms::allow_shared_memory(&device, 7, allowed) != cudaSuccess || ms::sm_count() != 100 + d) return 2;
    }
  for (int d : devices) std::printf("%d:%d:%d ", d, asked[d], counted[d]);
  return 0;
}
"""


@pytest.mark.skipif(CUDA is None or shutil.which("g++") is None, reason="needs g++ and the CUDA headers")
def test_every_device_is_asked_once(tmp_path):
    (tmp_path / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-x", "c++", "-I", str(CSRC), "-I", str(CUDA), str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main")], check=True)
    got = subprocess.run([str(tmp_path / "main")], check=True, capture_output=True, text=True).stdout.split()
    # (devices beyond those that are kept are asked each time; a refusal is not kept)
    assert got == ["0:7:1", "1:7:1", "63:7:1", "64:21:3"]


def test_no_kernel_keeps_one_devices_answer():
    for source in sorted(CSRC.glob("*.cu*")):
        assert not re.search(r"static[^;{]*\bcudaError_t\b[^;]*=\s*cudaFuncSetAttribute", source.read_text()), source.name


@pytest.mark.parametrize("source", ["gemm_f32.cu", "chunk_walk.cu"])
def test_no_multiprocessor_count_of_one_device(source):
    assert "cudaDevAttrMultiProcessorCount" not in (CSRC / source).read_text()
