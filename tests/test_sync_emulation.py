"""Barriers and warp operations of the block-wide searches, checked on the host: the device code itself, its
threads run as fibers in random orders (tests/cpp/cuda_emu.h). Every order has to keep the threads together and
give the sequential search's products (no GPU needed)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "shockhash_b200", "csrc")
CPP = os.path.join(ROOT, "tests", "cpp")


def run_emulated(source, tmp_path):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "emulated")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "-Xcompiler", "-Wno-attributes", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
                    "-I", CPP, "-I", str(tmp_path), "-x", "c++", os.path.join(CPP, source), "-o", exe],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr


def test_split_search_by_several_blocks(tmp_path):
    run_emulated("sync_split.cpp", tmp_path)
