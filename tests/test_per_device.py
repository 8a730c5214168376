"""What the kernels' launchers keep for a device they keep for each device (host code, no device needed)."""
import ctypes
import os
import subprocess

import pytest

_HERE = os.path.dirname(os.path.abspath(__file__))


def test_a_kernels_shared_memory_is_allowed_once_on_every_device(tmp_path):
    from torchless_rs_b200.csrc import build
    out = str(tmp_path / "libper_device.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.find_nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", os.path.dirname(build.__file__), "-I", cuda, "-o", out,
                    os.path.join(_HERE, "kernels", "per_device.cpp")], check=True, capture_output=True)
    lib = ctypes.CDLL(out)
    assert [lib.ask(1, 0, 0), lib.ask(1, 0, 0), lib.taken()] == [0, 0, 1]
    assert [lib.ask(1, 1, 0), lib.ask(1, 1, 0), lib.ask(1, 0, 0), lib.taken()] == [0, 0, 0, 2]
    assert [lib.ask(2, 1, 0), lib.taken()] == [0, 3]                       # another kernel
    assert lib.ask(2, 3, 1) != 0 and lib.ask(2, 3, 0) == 0                  # a failure is told and not kept
    assert lib.taken() == 5 and lib.ask(2, 3, 1) == 0
    assert [lib.ask(1, 64, 0), lib.ask(1, 64, 0), lib.taken()] == [0, 0, 7]  # beyond the table: asked each time


@pytest.mark.parametrize("source", ["gemm_split.cu", "attention_f32.cu", "latent_attention_tc.cu", "moe_tc.cu", "linear_recurrence.cu"])
def test_these_launchers_keep_no_attribute_for_the_whole_process(source):
    from torchless_rs_b200.csrc import build
    with open(os.path.join(os.path.dirname(build.__file__), source), encoding="utf-8") as f:
        text = f.read()
    assert "cudaFuncSetAttribute(" not in text and "tl_allow_smem<" in text
