"""The pages that a batch's images are copied into are mapped while the device
renders (csrc/host_pages.h): whole pages of the caller's array only, contents
kept, and nothing happens where that cannot be done."""

import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_populate_pages(tmp_path):
    exe = tmp_path / "host_pages"
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", os.path.join(HERE, "host_pages.cpp"), "-o", str(exe)],
                   check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert (run.returncode, run.stdout) == (0, "0\n"), run.stdout
