"""Range identifiers above 256 buckets: splitter counts at the edges of how they
are loaded and laid out (rounds of 2048, more or fewer than the table's 1024
cells), clustered, repeated and far-apart splitters, in the one-launch and the
staged form.  Against numpy.  Exact."""
import numpy as np
import pytest
import torch

import gpumultisplit_gb300 as gms
from gpu_util import host, to_dev
from gpumultisplit_gb300 import datagen

pytestmark = pytest.mark.gpu


def _splitters(kind, B, rng):
    if kind == "uniform":
        s = rng.integers(0, 1 << 32, B)
    elif kind == "clustered":  # nearly all in one cell of the table
        s = (1 << 31) + rng.integers(0, 1 << 20, B)
    elif kind == "repeated":
        s = rng.integers(0, 97, B) * 44_000_000
    else:  # the two ends
        s = np.concatenate([np.arange(B // 2), (1 << 32) - 1 - np.arange(B - B // 2)])
    return np.sort(s).astype(np.uint32)


@pytest.mark.parametrize("B", [257, 300, 1023, 1024, 1025, 2047, 2048, 2049, 4096, 8191, 8192])
@pytest.mark.parametrize("kind", ["uniform", "clustered", "repeated", "ends"])
def test_splitter_layouts(gms_lib, B, kind):
    rng = np.random.default_rng(B)
    spl = _splitters(kind, B, rng)
    d_spl = datagen.from_u32(spl, "cuda")
    for n in (9001, 2_700_003):
        keys = datagen.as_u32(datagen.uniform_u32(n, B))
        keys[: min(n, 2 * B)] = np.resize(np.concatenate([spl, spl - 1]), min(n, 2 * B))  # on and just below splitters
        ids = np.searchsorted(spl, keys, side="right").astype(np.int64) - 1
        ids[ids < 0] = B - 1
        order = np.argsort(ids, kind="stable")
        dk, dv = to_dev(keys), to_dev(np.arange(n, dtype=np.uint32))
        ok, ov = torch.zeros_like(dk), torch.zeros_like(dv)
        ctx = gms.multisplit_context(B)
        gms.multisplit_allocate_key_value(n, ctx)
        offs = gms.multisplit_key_value(dk, dv, ok, ov, n, ctx, gms.range_bucket(d_spl), True)
        np.testing.assert_array_equal(host(ok), keys[order])
        np.testing.assert_array_equal(host(ov), order.astype(np.uint32))
        cnt = np.bincount(ids, minlength=B)
        assert offs == [int(x) for x in np.cumsum(cnt) - cnt]
        hist = torch.zeros(B, dtype=torch.int32, device="cuda")
        gms.multisplit_histogram(dk, n, hist, B, gms.range_bucket(d_spl))
        np.testing.assert_array_equal(hist.cpu().numpy(), cnt)
