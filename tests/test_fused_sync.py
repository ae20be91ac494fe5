"""How the blocks of a one-launch call meet, and when the stages take its place
(tests/cpp/fused_sync_test.cu), on the host."""
import subprocess
from pathlib import Path

from gpumultisplit_gb300 import build as gbuild

ROOT = Path(__file__).resolve().parent.parent


def test_forms_and_refusals(tmp_path):
    exe = tmp_path / "fused_sync_test"
    subprocess.run([gbuild.nvcc_path(), *gbuild.ARCH_FLAGS, "-std=c++17", "-I", str(ROOT / "include"), "-I",
                    str(ROOT / "gpumultisplit_gb300" / "csrc"), str(ROOT / "tests" / "cpp" / "fused_sync_test.cu"),
                    "-o", str(exe)], check=True, stdout=subprocess.DEVNULL, stderr=subprocess.DEVNULL)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
