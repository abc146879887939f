"""What the compiler reports of the drop-in's kernels: no register spills, and
no structs passed through local memory (their stack frame holds the records of
the reference form's call, 40 bytes)."""
import os
import re
import subprocess

from kraken_3_gpu_b200 import build

CSRC = os.path.join(os.path.dirname(os.path.abspath(build.__file__)), "csrc")


def test_step_kernels_neither_spill_nor_pass_structs_in_memory(tmp_path):
    flags = [f for f in build.NVCC_FLAGS if f not in ("-shared", "-Xcompiler", "-fPIC")]
    out = subprocess.run([build.nvcc(), *flags, "-Xptxas=-v", "-c", "-o", str(tmp_path / "w.o"), "kr_world.cu"],
                         cwd=CSRC, capture_output=True, text=True, check=True)
    seen = 0
    for name, frame, stores, loads in re.findall(
            r"Function properties for (\S+)\s+(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads",
            out.stdout + out.stderr):
        if "step_kernel" in name:
            seen += 1
            assert int(stores) == int(loads) == 0 and int(frame) <= 64, (name, frame, stores, loads)
    assert seen == 2
