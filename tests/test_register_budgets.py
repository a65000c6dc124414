"""Kernels whose grids are sized for a number of CTAs per SM keep within the registers that leaves them (the compiler says; no GPU needed)."""
import importlib.util
import os
import re
import subprocess

from cera_b200 import types

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _registers(source, tmp_path):
    spec = importlib.util.spec_from_file_location("cera_b200_build", os.path.join(ROOT, "cera_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    cmd = [build.nvcc()] + build.ARCH + build.COMMON + ["-Xptxas", "-v", "-c", os.path.join(build.CSRC, source), "-o", str(tmp_path / "o.o")]
    text = subprocess.run(cmd, capture_output=True, text=True, check=True).stderr
    return re.findall(r"Compiling entry function '(\w+)'.*?Used (\d+) registers", text, re.S)


def test_ctas_of_a_decode_product_fit_an_sm(tmp_path):
    used = {tuple(map(int, re.search(r"gemv_rows_kernelILi(\d+)ELi\d+ELb(\d)E", name).groups())): int(r)
            for name, r in _registers("gemv_rows.cu", tmp_path) if "gemv_rows_kernel" in name}
    assert len(used) == 12  # six formats, the column quantized before or by the kernel
    for (fmt, forms), r in used.items():
        ctas = 1 if (fmt, forms) == (types.Q8_0, 1) else 2
        assert r * 256 * ctas <= 65536, (fmt, forms, r)
