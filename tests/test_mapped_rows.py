"""CPU test of the mapped host rows: counted over sessions, and never unmapped under a copy that shares their pages."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("sanitizer", ["undefined,address", "thread"])
def test_no_page_is_unmapped_under_a_copy(tmp_path, sanitizer):
    exe = str(tmp_path / "mapped_rows")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-fsanitize=" + sanitizer,
                        os.path.join(ROOT, "tests", "cpp", "mapped_rows.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout + out.stderr
