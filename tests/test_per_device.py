"""What the host remembers of kernels and devices is the device's own, and a choice is asked for the device of the operands."""
import os
import subprocess

import torch

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nanorlhf_b200", "csrc")
PROGRAM = r"""
#include "per_device.h"
static int device = 0, asked = 0;
static cudaError_t answer = cudaSuccess;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { ++asked; return answer; }
int main() {
  static nrl::PerDevice<int> n;
  static nrl::PerDevice<bool> done;
  const void* kernel = nullptr;
  auto asks = [&](int d, bool ok) { device = d; asked = 0; return (nrl::allow_smem(done, kernel, 1) == cudaSuccess) == ok ? asked : -1; };
  for (int d = 0; d < 64; ++d) { device = d; if (n.here() != 0) return 1; n.here() = d + 1; }
  for (int d = 0; d < 64; ++d) { device = d; if (n.here() != d + 1) return 2; }
  device = 64; n.here() = 9; if (n.here() != 0) return 3;             // not remembered
  if (asks(0, true) != 1 || asks(0, true) != 0 || asks(1, true) != 1 || asks(0, true) != 0 || asks(1, true) != 0 || asks(70, true) != 1 || asks(70, true) != 1) return 4;
  answer = cudaErrorInvalidValue;
  if (asks(2, false) != 1 || asks(2, false) != 1 || asks(1, true) != 0) return 5;
  return 0;
}
"""


def test_values_are_the_devices_own(tmp_path):
    from nanorlhf_b200.csrc.build import CUDA_HOME
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", f"-I{CUDA_HOME}/include", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_choices_are_asked_for_the_operands_device(monkeypatch):
    from nanorlhf_b200 import ops
    from nanorlhf_b200.ops import gemm
    asked = []

    class Ext:
        def gemm_tc_auto_splits(self, M, N, K, device):
            asked.append(device)
            return 2 if len(asked) > 1 else 1

    monkeypatch.setattr(ops, "use_native", lambda t: True)
    monkeypatch.setattr(gemm._native_mod, "ext", Ext)
    monkeypatch.setattr(torch.Tensor, "get_device", lambda t: 3)
    monkeypatch.setattr(gemm, "gemm", lambda a, b, **kw: torch.zeros(a.shape[0], b.shape[1]))
    x, w = torch.zeros(16, 8, dtype=torch.bfloat16), torch.zeros(8, 8, dtype=torch.bfloat16)
    assert gemm.linears(x, [w, torch.zeros(16, 8, dtype=torch.bfloat16)], [None, None]) is None
    assert gemm.swiglu_linears(x, (w, None, None), (w, None, None)) is None
    gemm.sum_gemms([x, x], [w, w])
    assert len(asked) == 4 and set(asked) == {3}
