"""Ranks that come from shared-memory atomics: the host test of the repair, and
on the GPU every way a warp ranks its keys (atomics, one or two frequent
buckets, ballots) at every bucket count that uses them, partial tiles included,
against numpy's stable argsort.  Exact."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from gpumultisplit_gb300 import build as gbuild
from gpumultisplit_gb300 import datagen

ROOT = Path(__file__).resolve().parent.parent


def test_repair_on_the_host(tmp_path):
    exe = tmp_path / "order_test"
    subprocess.run([gbuild.nvcc_path(), *gbuild.ARCH_FLAGS, "-std=c++17", "-I", str(ROOT / "include"), "-I",
                    str(ROOT / "gpumultisplit_gb300" / "csrc"), str(ROOT / "tests" / "cpp" / "order_test.cu"), "-o",
                    str(exe)], check=True, stdout=subprocess.DEVNULL, stderr=subprocess.DEVNULL)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


def _keys(kind, n, logb, rng):
    """Bucket ids in the top logb bits, low bits random so that order shows."""
    B = 1 << logb
    u = rng.integers(0, B, n)
    ids = {
        "uniform": u,
        "one": np.full(n, B - 1),
        "two": np.where(np.arange(n) % 2, 1, B - 2),
        "half": np.where(rng.random(n) < 0.5, 3 % B, u),
        "most": np.where(rng.random(n) < 0.9, 0, u),
        "three": rng.integers(0, 3, n),
        "four_far": rng.integers(0, 4, n) * (B // 4),
        "runs": (np.arange(n) // 37) % B,
        "warps": np.where((np.arange(n) // 512) % 2, u, 5 % B),       # crowded and plain warps in one tile
        "late": np.where(np.arange(n) % 512 < 32, u, 2 % B),          # first slot says nothing of the rest
        "early": np.where(np.arange(n) % 512 < 32, 2 % B, u),
    }[kind].astype(np.uint64)
    low = rng.integers(0, 1 << (32 - logb), n).astype(np.uint64)
    return ((ids << np.uint64(32 - logb)) | low).astype(np.uint32), ids.astype(np.int64)


KINDS = ["uniform", "one", "two", "half", "most", "three", "four_far", "runs", "warps", "late", "early"]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("logb", [4, 5, 6, 7, 8])
def test_every_way_to_rank(gms_lib, kind, logb):
    import torch

    import gpumultisplit_gb300 as gms
    from gpu_util import host, to_dev

    rng = np.random.default_rng(logb * 100 + KINDS.index(kind))
    B = 1 << logb
    # one tile, a partial one, and three stages (past the one-launch sizes)
    for n in (4096, 4096 + 700, 33, 3_000_019):
        keys, ids = _keys(kind, n, logb, rng)
        order = np.argsort(ids, kind="stable")
        dk, dv = to_dev(keys), to_dev(np.arange(n, dtype=np.uint32))
        for pairs in (False, True):
            for ident in (gms.delta_bucket(), gms.range_bucket(_splitters(B))):
                ok, ov = torch.zeros_like(dk), torch.zeros_like(dv)
                ctx = gms.multisplit_context(B)
                if pairs:
                    gms.multisplit_allocate_key_value(n, ctx)
                    gms.multisplit_key_value(dk, dv, ok, ov, n, ctx, ident)
                    np.testing.assert_array_equal(host(ov), order.astype(np.uint32))
                else:
                    gms.multisplit_allocate_key_only(n, ctx)
                    gms.multisplit_key_only(dk, ok, n, ctx, ident)
                np.testing.assert_array_equal(host(ok), keys[order])
                assert gms.read_device_error(ctx) == 0


def _splitters(B):
    """B equal ranges as splitters: the same buckets as delta."""
    return datagen.from_u32((np.arange(B, dtype=np.uint64) << np.uint64(32)) // np.uint64(B), "cuda")
