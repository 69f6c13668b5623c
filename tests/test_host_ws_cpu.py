"""Sampling from host logits: a call that fails half-way (host_ws.h, over a model of the CUDA runtime) spoils no later one."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))


def test_the_call_after_a_failed_one_is_right(tmp_path):
    exe = str(tmp_path / "host_ws")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-fsanitize=address,undefined", "-I", os.path.join(CUDA, "include"),
                           os.path.join(HERE, "host_ws_check.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert int(r.stdout) > 100
