"""The window filter's C entry with a buffer that its init refused (no GPU needed)."""
import os
import subprocess

from wema_b200 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_refused_window(tmp_path):
    lib = _build.build_cuda()
    exe = str(tmp_path / "window_refused")
    subprocess.run(["gcc", "-std=c11", "-O1", "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "c", "window_refused.c"), "-L", os.path.dirname(lib), "-lwema_cuda",
                    "-Wl,-rpath," + os.path.dirname(lib), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
