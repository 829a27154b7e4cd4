"""CPU test of how a batch is cut into sub-batches and where their slot ranges are noted: every part's marks lie inside arrays sized for
the batch, also where the tables of a residual batch make more than a thousand parts."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_marks_of_every_part_lie_inside(tmp_path):
    exe = str(tmp_path / "batch_parts")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-fsanitize=undefined,address", os.path.join(ROOT, "tests", "cpp", "batch_parts.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout + out.stderr
