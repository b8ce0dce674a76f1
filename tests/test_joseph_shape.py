"""The kernels that the host chooses for the scans of test_joseph_lines_gpu.py, on
the CPU: together they reach the line projector with several windows, its
refusal (the slab projector), and the backprojector's lines with and without
runs."""
import os
import subprocess

from fdk_cuda_impl_b200.geometry import CircularScan
from tests.test_joseph_lines_gpu import CASES

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "fdk_cuda_impl_b200")


def test_kernels_chosen(ykb_lib, tmp_path):
    out = str(tmp_path / "joseph_shape_test")
    objects = [os.path.join(PKG, "_build", f + ".o") for f in ("joseph_fp_lines.cu", "ykb_geometry.cpp")]
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(PKG, "csrc"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "joseph_shape_test.cpp"), *objects, "-o", out,
                    "-L/usr/local/cuda/lib64", "-lcudart_static", "-lpthread", "-ldl", "-lrt"], check=True)
    text = ""
    for views, nu, nv, pu, pv, n, vox, flipped in CASES:
        table = CircularScan(views, views, 500.0, 1000.0, nu, nv, pu, pv, start_angle_rad=0.05).views()
        if flipped:
            table["detS"][:, :3] += (nv - 1) * table["detV"][:, :3]
            table["detV"][:, :3] *= -1
        text += " ".join(map(str, (views, nu, nv, *n, *vox, 0.4, -0.7, 0.2))) + "\n"
        text += " ".join(repr(float(f)) for f in table.view("f4").ravel()) + "\n"
    res = subprocess.run([out], input=text, capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stderr
    chosen = [tuple(map(int, line.split())) for line in res.stdout.splitlines()]
    assert len(chosen) == len(CASES)
    windows = [w for _, w, _ in chosen]
    assert windows == [64, 64, 96, 64, 64, 128, 304, 256, 0]
    assert [r > 0 for r, _, _ in chosen] == [w > 0 for w in windows]
    assert [i for i, (_, _, runs) in enumerate(chosen) if runs] == [3, 4, 7]
