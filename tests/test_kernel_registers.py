"""The single-pass fluid kernels compile without register spills.

A spill in these kernels lands in the per-direction loops and their local
memory loads sit on the critical path: one of 8 bytes in the FP32 particle
variant once doubled its time (1.24 -> 2.67 ms per colloid step at 256^3).
The check compiles lbx_fused.cu with ptxas statistics (no GPU needed).
FP64 storage is exempt: its kernels run one CTA per SM at up to 255
registers and are not performance paths.
"""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def _ptxas_report(source):
    """Lines of the ptxas statistics of one source file, compiled as the build compiles it."""
    from lbcuda_b200 import build as B
    nvcc = B.nvcc()
    if not (os.path.isabs(nvcc) and os.path.exists(nvcc)) and shutil.which(nvcc) is None:
        pytest.skip("nvcc not available")
    cmd = [nvcc] + B.NVCC_FLAGS + B.FILE_FLAGS.get(source, []) + ["-Xptxas", "-v", "-c", os.path.join(B.CSRC, source),
                                                                  "-o", os.devnull]
    p = subprocess.run(cmd, capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-2000:]
    return p.stderr.splitlines()


@pytest.fixture(scope="module")
def fused_report():
    return _ptxas_report("lbx_fused.cu")


def test_lean_kernels_do_not_spill(fused_report):
    lines = fused_report
    cur = None
    checked = 0
    bad = []
    for line in lines:
        m = re.search(r"Compiling entry function '(\S+)'", line)
        if m:
            cur = m.group(1)
            continue
        m = re.search(r"(\d+) bytes spill stores, (\d+) bytes spill loads", line)
        if m and cur and "k_cg_lean" in cur:
            if "IdLi" in cur:  # FP64 storage instantiations
                continue
            checked += 1
            if int(m.group(1)) or int(m.group(2)):
                bad.append((cur, m.group(1), m.group(2)))
    assert checked >= 8, "no k_cg_lean instantiations found in the ptxas output"
    assert not bad, f"register spills in single-pass kernels: {bad}"


def test_march_kernels_do_not_spill():
    """The single-pass step of the two-density and D3Q27 models (lbx_fluid.cu), FP32 and 16-bit storage: 20 bytes of
    spills in its plane loop took 104 instead of 96 us at 96^3."""
    cur, spills = None, {}
    for line in _ptxas_report("lbx_fluid.cu"):
        m = re.search(r"Compiling entry function '(\S+)'", line)
        cur = m.group(1) if m else cur
        m = re.search(r"(\d+) bytes spill stores, (\d+) bytes spill loads", line)
        if m and cur and "k_cg_marchI" in cur and "k_cg_marchIdL" not in cur:
            spills[cur] = (int(m.group(1)), int(m.group(2)))
    assert len(spills) == 9 and set(spills.values()) == {(0, 0)}, spills


def test_two_role_kernels_launch_with_the_registers_they_share_out(fused_report):
    """k_cg_lean2 hands registers from its phase warps to its collision warps (setmaxnreg), which wait without a
    limit for any the launch did not allocate; every instance of this build is launched with the number that the
    two shares are made for."""
    cur, used = None, {}
    for line in fused_report:
        m = re.search(r"Compiling entry function '(\S+)'", line)
        cur = m.group(1) if m else cur
        m = re.search(r"Used (\d+) registers", line)
        if m and cur and "k_cg_lean2" in cur:
            used[cur] = int(m.group(1))
    assert len(used) >= 12 and set(used.values()) == {128}, used


def test_role_shares_are_checked_against_the_launch(tmp_path):
    """The host takes the two-role kernels only where the launch allocation holds both shares (56 + 200 for two
    threads): not with one register less, and not with a share on the wrong side of the allocation."""
    from lbcuda_b200 import build as B
    src = tmp_path / "roles.cpp"
    src.write_text('#include "lbx_roles.h"\n#include <cstdio>\n'
                   'int main() { for (int r = 24; r <= 255; ++r) if (lbx::role_regs_fit(r)) std::printf("%d\\n", r); }\n')
    exe = str(tmp_path / "roles")
    subprocess.run(["g++", "-std=c++17", "-I", B.CSRC, str(src), "-o", exe], check=True)
    fits = [int(v) for v in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()]
    assert fits == list(range(128, 201))
