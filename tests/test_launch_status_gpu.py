"""What an entry returns when a CUDA call fails."""
import subprocess

import pytest

from intent_b200.build import CSRC, NVCC_FLAGS, ROOT, _nvcc

pytestmark = pytest.mark.gpu

PROGRAM = """
#include <cuda_runtime.h>
#include <cstdio>
#include "common.cuh"
int main() {
  const cudaError_t e = cudaSetDevice(1 << 20);        // no such device
  const int status = ib200::cuda_status(e);
  std::printf("%d %d %d", int(e), status - INTENT_B200_ERR_CUDA, int(cudaPeekAtLastError()));
}
"""


def test_a_returned_error_does_not_linger(cuda_device, tmp_path):
    """The next call of the library must not report it a second time as its own."""
    source, binary = tmp_path / "status.cu", tmp_path / "status"
    source.write_text(PROGRAM)
    subprocess.run([_nvcc(), *NVCC_FLAGS, f"-I{CSRC}", f"-I{ROOT.parent / 'include'}", str(source), "-o", str(binary)],
                   check=True, capture_output=True)
    error, status, left = map(int, subprocess.run([str(binary)], check=True, capture_output=True, text=True).stdout.split())
    assert error != 0 and status == error
    assert left == 0
