"""The staged key form of the seed searches (SeedKey) against remix, on the host (no GPU needed)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_staged_keys_give_remix(tmp_path):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "seed_key")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "shockhash_b200", "csrc"), "-x", "cu",
                    os.path.join(ROOT, "tests", "cpp", "seed_key.cpp"), "-o", exe], check=True, capture_output=True, text=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
