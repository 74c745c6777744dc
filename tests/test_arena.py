"""The arena of a build's put-off tie repairs hands out ranges of mixed lengths
to thousands of warps at once; compile its reservation for the host and let
threads compete for it."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_ranges_do_not_overlap(tmp_path):
    exe = tmp_path / "arena_check"
    src = os.path.join(ROOT, "tests", "native", "arena_check.cpp")
    inc = os.path.join(ROOT, "falconnpp_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", f"-I{inc}", src, "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("ok")
