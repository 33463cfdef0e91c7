"""The library's host logic around the CUDA runtime (common.cu), compiled
against a fake runtime on host memory, so that failures and devices that no
test machine has can be played through without a GPU."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def _run(tmp_path, name, *args):
    exe = tmp_path / name
    src = os.path.join(ROOT, "imops_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", HERE, "-I", src, "-I", os.path.join(ROOT, "include"),
                    "-I", "/usr/local/cuda/include", "-x", "c++", os.path.join(HERE, name + ".cpp"),
                    os.path.join(src, "common.cu"), "-o", str(exe)], check=True, timeout=300)
    r = subprocess.run([str(exe), *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("name", ["host_working_sets", "host_side_streams"])
def test_host(tmp_path, name):
    _run(tmp_path, name)


@pytest.mark.parametrize("case", ["other_device", "slow_pinned_memory", "no_threads"])
def test_download(tmp_path, case):
    _run(tmp_path, "host_download", case)
