"""csrc/include/once_per_device.h: what is set up once on every device, and not once for the first device that comes."""
import os
import subprocess

INCLUDE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kv-cache-manager_b200", "csrc", "include")
CUDA = os.path.join(os.path.dirname(INCLUDE), "cuda")

PROGRAM = r"""
#include "once_per_device.h"
#include <cstdio>
int main() {
  kvcm::OncePerDevice once;
  int calls = 0;
  auto good = [&] { ++calls; return 0; };
  auto bad = [&] { ++calls; return 7; };
  const int rc[] = {once(0, bad), once(0, good), once(0, good), once(1, good), once(63, good), once(63, bad), once(64, good), once(64, good), once(-1, bad)};
  for (int r : rc) std::printf("%d ", r);
  std::printf("%d", calls);
}
"""


def test_every_device_is_set_up_and_a_failure_is_not_kept(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", INCLUDE, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "7 0 0 0 0 0 0 0 7 7"


def test_the_float32_and_split_k_products_set_their_limits_per_device():
    for name in ("gemm_f32.cu", "gemm_tcgen05_splitk.cu"):
        with open(os.path.join(CUDA, name)) as f:
            text = f.read()
        assert "cudaFuncSetAttribute" not in text and "allow_shared_memory(once" in text
