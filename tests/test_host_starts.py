"""The pinned words of calls that return bucket starts: the pool on the host with
a counting allocator, and on the GPU threads that come and go."""
import subprocess
import threading
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_pool_on_the_host(tmp_path):
    exe = tmp_path / "host_starts_test"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-O1", "-pthread", "-I",
                    str(ROOT / "gpumultisplit_gb300" / "csrc"), str(ROOT / "tests" / "cpp" / "host_starts_test.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


@pytest.mark.gpu
def test_threads_that_come_and_go(gms_lib):
    import numpy as np
    import torch

    import gpumultisplit_gb300 as gms
    from gpumultisplit_gb300 import datagen

    keys = datagen.uniform_u32(10007, 3, device="cuda")
    c = np.bincount((datagen.as_u32(keys) >> np.uint32(27)).astype(np.int64), minlength=32)
    want = [int(x) for x in np.cumsum(c) - c]
    ctx = gms.multisplit_context(32)
    gms.multisplit_allocate_key_only(keys.numel(), ctx)
    out = torch.empty_like(keys)
    got = []
    for _ in range(100):
        t = threading.Thread(target=lambda: got.append(
            gms.multisplit_key_only(keys, out, keys.numel(), ctx, gms.delta_bucket(), True)))
        t.start()
        t.join()
    assert got == [want] * 100
