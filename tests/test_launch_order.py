"""Launches behind a step's grouping kernel, stream by stream (the logic alone, on the CPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launch_order(tmp_path):
    exe = str(tmp_path / "order_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-o", exe, os.path.join(ROOT, "tests", "order_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
