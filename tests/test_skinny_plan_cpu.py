"""The plans of the projections of a few rows (csrc/skinny_plan.h), walked on the CPU over rows, outputs, K, blocks and SM counts."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_every_plan_stays_within_the_kernel_and_reads_k_in_order(tmp_path):
    exe = str(tmp_path / "walk")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(HERE, "..", "denograd_b200", "csrc"), os.path.join(HERE, "skinny_plan_walk.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
