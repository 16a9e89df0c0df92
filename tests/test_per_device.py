"""What the runtime keeps per device is set on every device of a process (csrc/per_device.h), and nothing in the kernels' launchers keeps such
a thing once per process."""
import glob
import os
import re
import subprocess

import pytest
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "infer_b200", "csrc")


def test_each_device_is_asked_once(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", exe, os.path.join(HERE, "per_device_check.cpp")], check=True)
    proc = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert proc.returncode == 0, proc.stdout


def test_launchers_keep_no_attribute_once_per_process():
    """A function-local static that stands for "done" or holds a runtime answer is a PerDevice."""
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(path) as f:
            src = f.read()
        for m in re.finditer(r"static (?:const )?(?:bool|int|cudaError_t) (\w+) *= *([^;]*);", src):
            tail = src[m.end():m.end() + 400]
            assert "cuda" not in m.group(2) and not re.search(r"if \(!%s\)" % m.group(1), tail), f"{os.path.basename(path)}: {m.group(0)}"


@pytest.mark.gpu
@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="one device")
@pytest.mark.parametrize("M", [1, 8, 200])
def test_the_32_bit_product_on_two_devices(M):
    from infer_b200 import ops
    g = torch.Generator().manual_seed(M)
    x, w = torch.randn(M, 512, generator=g), torch.randn(5000, 512, generator=g)
    got = []
    for d in ("cuda:0", "cuda:1"):
        with torch.cuda.device(d):
            got.append(ops.linear_plain(x.to(d), w.to(d)).cpu())
    assert torch.equal(*got)
