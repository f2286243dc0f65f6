"""The device status word and its host mirror."""

import ctypes
import os
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include "csrc/common.cuh"
__global__ void raise_kernel(int* status, int code) { kda::raise_status(status, code); }
extern "C" int raise_all(int* status, int code) {
    raise_kernel<<<4, 64>>>(status, code);
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
"""


def test_a_workspace_reports_its_first_failure_to_the_host_once(tmp_path):
    """Many threads raise the word of one workspace; the host reads and clears its mirror; threads of the same workspace that
    give up later must not set it again."""
    from experiment_swa_kda_b200 import build
    src, lib = tmp_path / "raise.cu", tmp_path / "raise.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc_path(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I" + os.path.join(ROOT, "experiment_swa_kda_b200"), str(src), "-o", str(lib)], check=True)
    fn = ctypes.CDLL(str(lib)).raise_all
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int]
    mirror = torch.zeros(1, dtype=torch.int32).pin_memory()
    words = torch.zeros(4, dtype=torch.int32, device="cuda:0")
    words.view(torch.int64)[1] = mirror.data_ptr()
    torch.cuda.synchronize()
    assert fn(words.data_ptr(), 53) == 0
    assert mirror.item() == 53 and words[0].item() == 53
    mirror.zero_()
    assert fn(words.data_ptr(), 54) == 0
    assert mirror.item() == 0 and words[0].item() == 53
