"""The classes of resident solve kernels that a handle loads and launches (res_class_mask in
ariel_b200/csrc/pcg.cuh) are those that its scenes can reach: compiled into a small host program and
checked over every FLUID count of grids up to 256^3; no GPU is needed."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_class_mask_is_what_the_grid_can_reach(tmp_path):
    from ariel_b200 import build as B
    exe = str(tmp_path / "res_classes")
    cmd = [B.nvcc()] + B.ARCH + ["-std=c++17", "-O2", "-ccbin", B.host_compiler(),
                                 "-I", os.path.join(ROOT, "ariel_b200", "csrc"),
                                 os.path.join(ROOT, "tests", "cpp", "res_classes.cu"), "-o", exe]
    subprocess.run(cmd, check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
