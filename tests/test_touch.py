"""The host threads that touch a download's pages ahead of its copies."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "axion-strings_gb300", "csrc")


def run(tmp_path, name):
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, os.path.join(HERE, name + ".cpp"), "-o", exe, "-pthread", "-ldl"],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    if r.stdout.startswith("skip"):
        pytest.skip("too few host threads")
    assert r.returncode == 0, r.stdout


def test_no_write_after_a_thread_could_not_be_created(tmp_path):
    run(tmp_path, "touch_threads")


def test_only_missing_pages_are_touched(tmp_path):
    run(tmp_path, "touch_resident")
