"""Bucket starts returned to the host: several threads at once, each on its own
stream and scratch, sizes of the one-launch and the three-stage form, and every
entry point that returns them.  Whole numbers: every comparison is exact."""
import threading

import numpy as np
import pytest
import torch

import gpumultisplit_gb300 as gms
from gpumultisplit_gb300 import datagen

pytestmark = pytest.mark.gpu


def _expected(keys, B):
    ids = (keys.astype(np.uint64) * np.uint64(B)) >> np.uint64(32)
    c = np.bincount(ids.astype(np.int64), minlength=B)
    return [int(x) for x in np.cumsum(c) - c]


@pytest.mark.parametrize("n", [5000, 700_001, 5_000_003])
def test_threads_get_their_own_offsets(gms_lib, n):
    """Eight threads call with different keys and bucket counts; none sees another's starts."""
    bad, jobs = [], []
    for i in range(8):
        B = (2, 7, 32, 256, 100, 64, 255, 16)[i]
        keys = datagen.uniform_u32(n + i, 70 + i, device="cuda")
        jobs.append((B, keys, torch.empty_like(keys), _expected(datagen.as_u32(keys), B)))
    torch.cuda.synchronize()

    def work(B, keys, out, want):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                ctx = gms.multisplit_context(B)
                gms.multisplit_allocate_key_only(keys.numel(), ctx)
                for _ in range(30):
                    got = gms.multisplit_key_only(keys, out, keys.numel(), ctx, gms.delta_bucket(), True)
                    if got != want:
                        bad.append((B, got[:4], want[:4]))
                c2 = gms.compaction_context()
                gms.compaction_allocate_key_only(keys.numel(), c2)
                zeros = int((keys & 1 == 0).sum())
                for _ in range(10):
                    if gms.compaction_key_only(keys, out, keys.numel(), c2, gms.mask_bucket(1)) != zeros:
                        bad.append(("compaction", B))
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            bad.append(repr(e))

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]


@pytest.mark.parametrize("n", [1, 3000, 4_000_001])
@pytest.mark.parametrize("widths", [(8, 0), (8, 8), (4, 8), (4, 4)])
def test_wide_offsets(gms_lib, n, widths):
    kb, vb = widths
    keys = datagen.uniform_u64(n, 3, device="cuda") if kb == 8 else datagen.uniform_u32(n, 3, device="cuda")
    vals = torch.arange(n, dtype=torch.int64 if vb == 8 else torch.int32, device="cuda") if vb else None
    out, vout = torch.empty_like(keys), torch.empty_like(vals) if vb else None
    ctx = gms.multisplit_context(64)
    gms.multisplit_wide_allocate(n, ctx, kb, vb)
    got = gms.multisplit_wide(keys, out, n, ctx, gms.delta_bucket(), vals, vout, True)
    top = (datagen.as_u64(keys) >> np.uint64(58)) if kb == 8 else (datagen.as_u32(keys) >> np.uint32(26))
    c = np.bincount(top.astype(np.int64), minlength=64)
    assert got == [int(x) for x in np.cumsum(c) - c]
