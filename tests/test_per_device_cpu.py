"""Shared memory beyond 48 KB is asked for once on every device of a process, not once a process (a stand-in for the CUDA runtime
counts the requests)."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tokasaurus_b200" / "csrc"
PROGRAM = r"""
#include "per_device.h"
#include <cstdio>
static int device = 0, requests = 0, fail = 0;
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
  requests++;
  return fail ? cudaErrorInvalidValue : cudaSuccess;
}
int main() {
  static tkb::SharedMemoryRequest ask;
  auto step = [&](int d, int f) {
    device = d, fail = f, requests = 0;
    int rc = ask({{(const void*)&device, 1}, {(const void*)&fail, 2}});
    printf("%d:%d ", rc, requests);
  };
  step(0, 0), step(0, 0), step(1, 0), step(0, 0), step(1, 0), step(2, 1), step(2, 0), step(2, 0), step(64, 0), step(64, 0);
}
"""


def test_every_device_is_asked_once(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = Path(nvcc).resolve().parent.parent / "include"
    if not (include / "cuda_runtime_api.h").is_file():
        pytest.skip("no CUDA headers")
    (tmp_path / "p.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", f"-I{include}", str(tmp_path / "p.cpp"), "-o", str(tmp_path / "p")], check=True)
    out = subprocess.run([str(tmp_path / "p")], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0:2", "0:0", "0:2", "0:0", "0:0", "1:1", "0:2", "0:0", "0:2", "0:2"]


def test_the_new_kernels_ask_by_device():
    for name in ("sgemm.cu", "decay_chunks.cu", "attention_rows_tc.cu"):
        text = (CSRC / name).read_text()
        assert "SharedMemoryRequest" in text and "static bool" not in text
