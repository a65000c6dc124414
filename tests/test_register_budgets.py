"""Kernels whose grids are sized for a number of CTAs per SM keep within the registers that leaves them (the compiler says; no GPU needed)."""
import importlib.util
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _registers(source, tmp_path):
    spec = importlib.util.spec_from_file_location("cera_b200_build", os.path.join(ROOT, "cera_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    cmd = [build.nvcc()] + build.ARCH + build.COMMON + ["-Xptxas", "-v", "-c", os.path.join(build.CSRC, source), "-o", str(tmp_path / "o.o")]
    text = subprocess.run(cmd, capture_output=True, text=True, check=True).stderr
    return re.findall(r"Compiling entry function '(\w+)'.*?Used (\d+) registers", text, re.S)


@pytest.mark.parametrize("source,kernel,threads,ctas,variants", [("gemv_rows.cu", "gemv_rows_kernel", 256, 2, 12)])
def test_ctas_of_a_decode_product_fit_an_sm(tmp_path, source, kernel, threads, ctas, variants):
    used = [int(r) for name, r in _registers(source, tmp_path) if kernel in name]
    assert len(used) == variants
    assert max(used) * threads * ctas <= 65536, used
