"""Kernels whose point is that a whole piece's rows are in registers, checked against what the compiler
reports: an array indexed at run time would lie in local memory instead."""
import importlib
import os
import re
import subprocess

import pytest

kb = importlib.import_module("kmeans_gb300.build")


@pytest.mark.parametrize("source,kernel", [("update.cu", "piece_sums_few_kernel")])
def test_no_local_memory(tmp_path, source, kernel):
    r = subprocess.run([kb.nvcc(), *kb.ARCH, *kb.COMMON, "-Xptxas=-v", "-c", os.path.join(kb.CSRC, source),
                        "-o", str(tmp_path / "o.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    frames = re.findall(r"Function properties for (\S*%s\S*)\s+(\d+) bytes stack frame, (\d+) bytes spill"
                        % kernel, r.stderr)
    assert frames and all(f[1:] == ("0", "0") for f in frames), frames
