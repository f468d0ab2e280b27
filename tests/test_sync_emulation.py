"""Barriers and warp operations of the block-wide searches, checked on the host: the device code itself, its
threads run as fibers in random orders (tests/cpp/cuda_emu.h). Every order has to keep the threads together and
give the sequential search's products (no GPU needed)."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

from conftest import unique_u64

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "shockhash_b200", "csrc")
CPP = os.path.join(ROOT, "tests", "cpp")


def run_emulated(source, tmp_path, *args):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "emulated")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "-Xcompiler", "-Wno-attributes", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
                    "-I", CPP, "-I", str(tmp_path), "-x", "c++", os.path.join(CPP, source), "-o", exe],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe, *args], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr


def test_split_search_by_several_blocks(tmp_path):
    run_emulated("sync_split.cpp", tmp_path)


def kernels_of(name, cuts):
    """The device code of a source file: without the parts [start, end) that launch kernels, which C++ cannot
    read, with dynamic shared memory from the emulation and plain copies for the asynchronous ones."""
    text = open(os.path.join(CSRC, name)).read()
    for start, end in cuts:
        i = text.index(start)
        text = text[:i] + (text[text.index(end, i):] if end else "")
    text = re.sub(r'asm volatile\("cp\.async\.cg[^;]*;[^;]*;', "memcpy(smem_dst, gsrc, 16);", text)
    text = re.sub(r'asm volatile\("cp\.async\.(commit|wait)[^;]*;[^;]*;', "", text)
    text = text.replace("extern __shared__ uint16_t rot_cells[];", "uint16_t *const rot_cells = (uint16_t *)emu::shared;")
    return text.replace("extern __shared__ __align__(16) uint8_t smem_raw[];", "uint8_t *const smem_raw = emu::shared;")


def test_leaf_searches(tmp_path, port):
    sh1 = kernels_of("shg_leaves.cu", [("int leaves_sh1_warps_per_block()", "")])
    sh2 = kernels_of("shg_leaves_sh2.cu", [("template <int MAXM, int MINB>\nvoid launch_v2(", "// ----"),
                                           ("template <int MAXM>\nvoid launch_block(", "")])
    (tmp_path / "leaves_sh1.inc").write_text(sh1 + "} // namespace shg\n")
    (tmp_path / "leaves_sh2.inc").write_text(sh2 + "} // namespace\n} // namespace shg\n")
    rng = np.random.default_rng(6)
    lines = []
    for kind, sizes in ((1, (22,)), (1, (1, 2, 9, 20, 16, 23)), (1, (25, 24)), (2, (64,)), (2, (57, 30, 64, 2, 9, 10, 48, 61, 63, 40)),
                        (2, (66,))):
        lines.append(f"{kind} {len(sizes)}")
        for m in sizes:
            keys = unique_u64(rng, m)
            seed, order, bits = port.sh1_leaf(keys) if kind == 1 else port.sh2_leaf(keys)
            bit = dict(zip(order.tolist(), bits.tolist()))
            lines.append(" ".join(str(v) for v in [m, seed, *keys.tolist(), *(bit[k] for k in keys.tolist())]))
    (tmp_path / "cases.txt").write_text("\n".join(lines) + "\n")
    run_emulated("sync_leaves.cpp", tmp_path, str(tmp_path / "cases.txt"))
