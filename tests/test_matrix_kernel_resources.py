"""CPU test of the compiled resources of the DP matrix kernels (nvcc
cross-compiles for sm_100a without a GPU): no form of them, the one of 16 rows
a lane included, keeps values in local memory."""
import os
import re
import subprocess

from test_kernel_resources import CSRC, _nvcc


def test_no_matrix_kernel_spills(tmp_path):
    import pytest
    from trajsimimeasures_b200 import build as B
    if not _nvcc():
        pytest.skip("nvcc is not available")
    cmd = [_nvcc()] + B.ARCH + B.FLAGS + ["-Xptxas=-v", "-c", "-I", B.INCLUDE, "-I", B.CSRC, "-o",
                                          str(tmp_path / "k.o"), os.path.join(CSRC, "tsm_k_matrix_fast.cu")]
    out = subprocess.run(cmd, capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-2000:]
    spills, cur = {}, None
    for line in (out.stdout + out.stderr).splitlines():
        m = re.search(r"Compiling entry function '(\S+)'", line)
        if m:
            cur = m.group(1)
        m = re.search(r"(\d+) bytes spill stores", line)
        if m and cur:
            spills[cur] = int(m.group(1))
    kernels = {k: v for k, v in spills.items() if "dp_matrix_kernel" in k}
    assert len(kernels) == 9, sorted(spills)  # three measures, 4, 8 and 16 rows
    assert not any(kernels.values()), kernels
