"""The bounded waits of the tensor-core kernels' warps (csrc/tc_ops.cuh): all lanes of a warp learn the same outcome, also where a wait
runs out for some of them only, and what the arriving thread had stored is there for every lane."""
import ctypes
import os
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_a_warp_agrees_on_every_wait(tmp_path):
    from infer_b200.csrc import build
    so = str(tmp_path / "wait_check.so")
    subprocess.run([build._find_nvcc()] + build.NVCC_FLAGS + ["-I", build.HERE, "-o", so, os.path.join(HERE, "wait_check.cu")], check=True,
                   capture_output=True, timeout=300)
    f = ctypes.CDLL(so).wait_check
    f.argtypes = [ctypes.c_void_p] * 2
    out = torch.full((5, 32), -2, dtype=torch.int32, device="cuda:0")
    assert f(out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert out.tolist() == [[v] * 32 for v in (0, 0, 0, 1, 7)]
