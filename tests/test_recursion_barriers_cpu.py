"""The L-BFGS kernels' shared-memory reductions, warp by warp on the CPU: their
results may not depend on which warp of a block runs ahead of the others
(emulated_block.cpp holds each warp back as long as its barriers allow)."""
import os
import re
import shutil
import subprocess

import pytest

TESTS = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(TESTS)
CSRC = os.path.join(ROOT, "packing_b200", "csrc")


def _kernel_text():
    """common.cuh and the L-BFGS kernels of lbfgs.cuh without their includes,
    the inline PTX replaced by the emulated operations."""
    common = open(os.path.join(CSRC, "common.cuh")).read()
    lbfgs = open(os.path.join(CSRC, "lbfgs.cuh")).read()
    kernels = lbfgs[lbfgs.index("// Two-loop recursion"):lbfgs.index("// One warp per canonical group")]
    text = common + kernels
    text = re.sub(r"^#include <.*$|^#include \"\.\./.*$|^#pragma once.*$", "", text, flags=re.M)
    text, n = re.subn(r'asm volatile\("redux\.sync\.max\.f32[^;]*;"[^;]*;', "r = warp_max(v);", text)
    assert n == 1
    text, n = re.subn(r'asm volatile\("bar\.sync 1, %0;"[^;]*;', "block_barrier(1, 32 * nw);", text)
    assert n == 1 and "asm" not in text
    # what each thread got from the reduction on either side of the recursion
    for at, value in (("bool fresh = false;", "{ys, yy, gmax, pc}"), ("if (prm.has_max_step &&", "{gtd[0], pc[0]}")):
        head, tail = text.split("void pk_lbfgs_iterate_kernel", 1)
        assert tail.count(at) == 1
        text = head + "void pk_lbfgs_iterate_kernel" + tail.replace(at, f"record({value}); {at}")
    header = open(os.path.join(ROOT, "include", "packb200.h")).read()
    return header + text


@pytest.fixture(scope="module")
def emulator(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("emulated")
    inc, exe = d / "kernels.inc", d / "emulated_block"
    inc.write_text(_kernel_text())
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-ffp-contract=off", "-w", f'-DKERNELS_INC="{inc}"', "-o", str(exe),
                        os.path.join(TESTS, "emulated_block.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return str(exe)


# N elements, threads: warps that own none of them (1 of 2; 3 of 8; 7 of 8), all
# owning one group (8 of 8), and more groups than warps
@pytest.mark.parametrize("N,threads", [(100, 64), (128, 64), (603, 256), (30, 256), (1024, 256), (300, 64), (1153, 256)])
def test_results_do_not_depend_on_which_warp_runs_ahead(emulator, N, threads):
    for m in (1, 3) + ((1030,) if N in (100, 603) else ()):   # 1030: the maxima have no room beside the sums
        r = subprocess.run([emulator, str(N), str(m), str(threads)], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
