"""The persistent decode kernel's unit layout (persist_plan.h) walked on the CPU: every unit shape that has a plan, and the plans of
all matrices of the two configurations, give the product exactly and read nothing outside the unit or the digits."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
MATRICES = ((1152, 1536), (1024, 1152), (1152, 6912), (6912, 1152), (640, 1536), (1024, 640), (640, 2048), (2048, 640))


def test_every_unit_multiplies_exactly(tmp_path):
    exe = str(tmp_path / "units")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", os.path.join(HERE, "persist_plan_check.cpp"), "-o", exe])
    r = subprocess.run([exe] + [str(v) for m in MATRICES for v in m], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert int(r.stdout) > 100
