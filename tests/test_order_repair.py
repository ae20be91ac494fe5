"""The postscan's check of a tile's order and its repair, on tiles whose runs
come in any order (tests/cpp/order_repair_test.cu).  On this chip the ranks come
back in order, so calls never reach the repair by themselves."""
import subprocess

import pytest

from test_dropin import BUILD, ROOT, _nvcc


def _build():
    from gpumultisplit_gb300 import build as gbuild

    BUILD.mkdir(parents=True, exist_ok=True)
    exe, src = BUILD / "order_repair_test", ROOT / "tests" / "cpp" / "order_repair_test.cu"
    deps = [src] + sorted((ROOT / "gpumultisplit_gb300" / "csrc").glob("*.cuh"))
    if not exe.exists() or any(exe.stat().st_mtime <= p.stat().st_mtime for p in deps):
        subprocess.run([_nvcc(), *gbuild.ARCH_FLAGS, "-O2", "-std=c++17", "-I", str(ROOT / "include"), "-I",
                        str(ROOT / "gpumultisplit_gb300" / "csrc"), str(src), "-o", str(exe)], check=True)
    return exe


@pytest.mark.gpu
def test_any_order_becomes_the_input_order():
    r = subprocess.run([str(_build())], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
