"""What the compiler reports for kernels whose register budget is tight (CPU only: nvcc cross-compiles)."""
import os
import re
import shutil
import subprocess

import pytest

from nlchains_gb300 import builder


def spills(source, tmp_path):
    """Spill bytes (stores, loads) of every kernel of a translation unit, by mangled name."""
    if not (os.path.exists(builder.NVCC) or shutil.which("nvcc")):
        pytest.skip("no nvcc")
    cmd = builder._cu_cmd(os.path.join(builder.CSRC, source), str(tmp_path / "o.o"))
    text = subprocess.run(cmd + ["-Xptxas", "-v"], capture_output=True, text=True, check=True).stderr
    found = {}
    for part in text.split("Compiling entry function '")[1:]:
        m = re.search(r"(\d+) bytes spill stores, (\d+) bytes spill loads", part)
        found[part.split("'")[0]] = (int(m.group(1)), int(m.group(2)))
    return found


def test_transform_split_step_has_a_form_without_integer_operations(tmp_path):
    """The DNLS transform kernel runs in 64 registers, for which the integer-pipe additions are too many:
    ensembles of few warps have instantiations without them, warp teams and blocks."""
    kernels = {k: v for k, v in spills("nlc_dnls.cu", tmp_path).items() if "dnls_move_kernel" in k}
    light = [v for v in kernels.values() if v[0] <= 100 and v[1] <= 150]
    assert len(light) == 2, kernels
