"""The scan of the prescan's rows: the status words it uses are words that the
prescan resets (a build that breaks this does not compile), and on the GPU its
results and its bounded wait (tests/cpp/scan_rows_test.cu)."""
import subprocess
from pathlib import Path

import pytest

from gpumultisplit_gb300 import build as gbuild

ROOT = Path(__file__).resolve().parent.parent
FLAGS = [*gbuild.ARCH_FLAGS, "-std=c++17", "-I", str(ROOT / "include"), "-I", str(ROOT / "gpumultisplit_gb300" / "csrc")]


@pytest.mark.parametrize("scan_ipt,compiles", [(16, True), (32, False)])
def test_status_words_cover_the_rows(tmp_path, scan_ipt, compiles):
    src = tmp_path / "t.cu"
    src.write_text('#include "scan_kernels.cuh"\n')
    r = subprocess.run([gbuild.nvcc_path(), *FLAGS, f"-DGMS_SCAN_IPT={scan_ipt}", "-c", str(src), "-o",
                        str(tmp_path / "t.o")], capture_output=True, text=True)
    assert (r.returncode == 0) == compiles, r.stderr
    assert compiles or "status word" in r.stderr + r.stdout


@pytest.mark.gpu
def test_results_and_bounded_wait(tmp_path):
    exe = tmp_path / "scan_rows_test"
    subprocess.run([gbuild.nvcc_path(), *FLAGS, str(ROOT / "tests" / "cpp" / "scan_rows_test.cu"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
