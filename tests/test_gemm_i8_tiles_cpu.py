"""The integer GEMM's tile arithmetic (gemm_i8_tiles.h) walked on the CPU over every matrix size that the operators take
and up to 32768 rows: every tile of every plan lies inside the product and is the one that exact division gives."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
K = (256, 640, 1024, 1152, 2048, 6912)
N = K + (262144,)


def test_every_tile_of_every_plan(tmp_path):
    exe = str(tmp_path / "tiles")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", os.path.join(HERE, "gemm_i8_tiles_check.cpp"), "-o", exe])
    r = subprocess.run([exe] + [str(v) for v in K + (0,) + N], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert int(r.stdout.split()[0]) > 1000000
