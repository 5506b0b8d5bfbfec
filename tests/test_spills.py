"""The multi-RHS kernels keep their sums and operands in registers: ptxas reports no spill for the
adjoint with its value gradient at any width.  Compiles gs_spmm.cu (some 20 s)."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "gpu_spmv_b200", "csrc")


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
def test_adjoint_kernels_do_not_spill(tmp_path):
    r = subprocess.run(["nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a",
                        "-I", os.path.join(CSRC, "..", "..", "include"),
                        "--expt-relaxed-constexpr", "-diag-suppress", "177", "-Xptxas", "-v", "-c",
                        os.path.join(CSRC, "gs_spmm.cu"), "-o", str(tmp_path / "o")],
                       capture_output=True, text=True, check=True)
    found = {}
    for name, spilled in re.findall(
            r"Compiling entry function '\w*k_k1_mmI(\w+?)ELb1E\w*'.*?(\d+) bytes spill stores",
            r.stderr, re.S):
        found[name] = int(spilled)
    assert set(found) == {t + "Li" + k for t in "df" for k in ("1", "2", "4", "8", "16", "32")}
    assert not any(found.values()), found
