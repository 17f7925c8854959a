"""An allocation that fails inside the GKR prover is reported as what it is: an out-of-memory or device
status with a message of its own, and (seen with a device only: without a driver every call fails alike) no
error left pending for the next launch's check to find. A host program links the prover's objects with an
allocator that always fails, so nothing is ever launched."""
import subprocess

import pytest

PROGRAM = r"""
#define stream_alloc unused_stream_alloc
#include "runtime.cu"
#undef stream_alloc
#include <cstring>
#include "gkr.cuh"
namespace cs {
cudaError_t g_failed = cudaSuccess;
cudaError_t stream_alloc(void** ptr, size_t, cudaStream_t) {
  return g_failed = cudaMalloc(ptr, (size_t)1 << 60);  // more than any device has
}
}  // namespace cs
int main() {
  cs::GkrInput in;
  in.kind = CS_GKR_GRAND_PRODUCT;
  in.n_vars = 3;
  uint32_t word = 0, chan[9] = {0};
  for (int k = 0; k < 4; k++) in.den[k] = &word;
  std::vector<uint64_t> out;
  cs::set_error("an earlier failure");
  const cs_status s = cs::gkr_prove_on_device({in}, chan, out, nullptr);
  const cudaError_t pending = cudaPeekAtLastError();
  const cs_status want = cs::g_failed == cudaErrorMemoryAllocation ? CS_ERR_OOM : CS_ERR_DEVICE;
  std::printf("status %d (%d) pending %d message %s\n", (int)s, (int)want, (int)pending, cs::last_error());
  const bool cleared = pending == cudaSuccess || want != CS_ERR_OOM;
  return s == want && cleared && std::strstr(cs::last_error(), "gkr_prove_batch") ? 0 : 1;
}
"""


def _run(tmp_path) -> subprocess.CompletedProcess:
    from proving_gb300 import build
    build.build()
    src, exe = tmp_path / "alloc.cu", tmp_path / "alloc"
    src.write_text(PROGRAM)
    cmd = [build.nvcc(), build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", f"-I{build.CSRC}", f"-I{build.INCLUDE}",
           str(src), str(build.BUILD / "gkr_prove.o"), str(build.BUILD / "gkr.o"), "-cudart", "static", "-o", str(exe)]
    subprocess.run(cmd, check=True, capture_output=True, text=True)
    return subprocess.run([str(exe)], capture_output=True, text=True)


def test_failed_allocation_is_reported(tmp_path):
    r = _run(tmp_path)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
def test_failed_allocation_is_cleared(tmp_path):
    r = _run(tmp_path)
    assert r.returncode == 0 and "status 2 (2) pending 0 " in r.stdout, r.stdout + r.stderr
