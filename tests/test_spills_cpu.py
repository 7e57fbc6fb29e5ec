"""Register spills of the closure's kernels, from the assembler's report: all of
L1 is given to shared memory there, so a spilled word comes back from L2.  The
lattice inference kernel at its 80 registers needs 24 bytes a thread (the next
tile's raw inputs are held across the matrix steps); 72 bytes made a refresh of
the correction 18% slower."""
import os
import re
import shutil
import subprocess

import pytest

from entropicthreadsafe_b200 import build

pytestmark = pytest.mark.skipif(not (os.path.exists(build.NVCC) or shutil.which(build.NVCC)), reason="needs nvcc")


def test_closure_kernels_spill_no_more(tmp_path):
    cmd = [build.NVCC, *build.CFLAGS, "-cubin", "-o", str(tmp_path / "closure.cubin"), os.path.join(build.CSRC, "closure.cu")]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    spills = {m.group(1): int(m.group(2)) for m in re.finditer(
        r"Function properties for (\S+)\n.*?(\d+) bytes spill stores", res.stderr)}
    lattice = [v for k, v in spills.items() if "infer_kernel" in k and "LatticeSrc" in k]
    train = [v for k, v in spills.items() if "train_kernel" in k]
    assert len(lattice) == 1 and len(train) == 1
    assert lattice[0] <= 24 and train[0] == 0, spills
