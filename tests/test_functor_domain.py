"""User functors with a limited key domain: evaluated on the input's keys only,
whatever a tile's unused slots hold (tests/cpp/functor_domain_test.cu)."""
import subprocess

import pytest

from test_dropin import BUILD, ROOT, _nvcc


def _build():
    from gpumultisplit_gb300 import build as gbuild

    lib = gbuild.build()
    BUILD.mkdir(parents=True, exist_ok=True)
    exe, src = BUILD / "functor_domain_test", ROOT / "tests" / "cpp" / "functor_domain_test.cu"
    deps = [src, lib] + list((ROOT / "include" / "gpumultisplit").rglob("*.cuh"))
    if not exe.exists() or any(exe.stat().st_mtime <= p.stat().st_mtime for p in deps):
        subprocess.run([_nvcc(), *gbuild.ARCH_FLAGS, "-O2", "-std=c++17", "-I", str(ROOT / "include"),
                        "-I", str(ROOT / "include" / "gpumultisplit"), "-I", str(ROOT / "gpumultisplit_gb300" / "csrc"),
                        str(src), "-L", str(lib.parent), "-lgpumultisplit", "-Xlinker", "-rpath", "-Xlinker",
                        str(lib.parent), "-o", str(exe)], check=True)
    return exe


@pytest.mark.gpu
def test_no_key_outside_the_domain():
    r = subprocess.run([str(_build())], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
