"""Identifiers whose division by a call's own number runs as a multiplication:
divisors and bucket counts at the edges of the reciprocal's cases, keys at the
edges of every quotient, against integer division on the host.  Exact."""
import numpy as np
import pytest
import torch

import gpumultisplit_gb300 as gms
from gpu_util import host, to_dev
from gpumultisplit_gb300 import datagen

pytestmark = pytest.mark.gpu

DIVISORS = [1, 2, 3, 5, 7, 10, 641, 1000003, (1 << 16) - 1, 1 << 16, (1 << 16) + 1, (1 << 31) - 1, 1 << 31,
            (1 << 31) + 1, (1 << 32) - 2, (1 << 32) - 1]


def _keys(d, n, seed):
    """Random keys, the two ends, and both sides of multiples of d."""
    rnd = datagen.as_u32(datagen.uniform_u32(n, seed)).astype(np.uint64)
    k = np.arange(n, dtype=np.uint64) % np.uint64((1 << 32) // d + 1)
    near = k * np.uint64(d) + (np.arange(n, dtype=np.uint64) % np.uint64(3)) - np.uint64(1)
    keys = np.where(np.arange(n) % 2 == 0, rnd, near & np.uint64(0xFFFFFFFF)).astype(np.uint32)
    keys[:4] = (0, 1, 0xFFFFFFFF, 0xFFFFFFFE)
    return keys


def _check(keys, B, ident, ids, with_values):
    n = keys.size
    ctx = gms.multisplit_context(B)
    dk, ok = to_dev(keys), to_dev(np.zeros(n, np.uint32))
    order = np.argsort(ids, kind="stable")
    if with_values:
        dv, ov = to_dev(np.arange(n, dtype=np.uint32)), to_dev(np.zeros(n, np.uint32))
        gms.multisplit_allocate_key_value(n, ctx)
        gms.multisplit_key_value(dk, dv, ok, ov, n, ctx, ident)
        np.testing.assert_array_equal(host(ov), order.astype(np.uint32))
    else:
        gms.multisplit_allocate_key_only(n, ctx)
        gms.multisplit_key_only(dk, ok, n, ctx, ident)
    np.testing.assert_array_equal(host(ok), keys[order])


@pytest.mark.parametrize("B", [2, 3, 100, 255, 256, 1000, 65536])
@pytest.mark.parametrize("d", DIVISORS)
def test_division_and_remainder(gms_lib, d, B):
    n = 20011
    keys = _keys(d, n, d % 1000 + B)
    ids = ((keys.astype(np.uint64) // np.uint64(d)) % np.uint64(B)).astype(np.int64)
    _check(keys, B, gms.delta_func(d), ids, with_values=B % 2 == 0)
    hist = torch.zeros(B, dtype=torch.int32, device="cuda")
    gms.multisplit_histogram(to_dev(keys), n, hist, B, gms.delta_func(d))
    np.testing.assert_array_equal(hist.cpu().numpy(), np.bincount(ids, minlength=B))


@pytest.mark.parametrize("B", [7, 100, 256, 1000])
@pytest.mark.parametrize("n", [20011, 3_000_017])
@pytest.mark.parametrize("lower,scale", [(0, 1.0), (1 << 20, 1.0), (12345, 3.7), (0, 1e-3), (5, 1e30)])
def test_even_float_wraps(gms_lib, B, n, lower, scale):
    """Bins past the last one, keys below the lower level, and a scale that saturates."""
    keys = datagen.as_u32(datagen.uniform_u32(n, B))
    keys[:3] = (0, lower, 0xFFFFFFFF)
    inv = np.float32(B / 2.0**32 * scale)
    x = (keys - np.uint32(lower)).astype(np.float32) * inv
    q = np.where(x >= np.float32(2.0**32), np.float64(2**32 - 1), np.floor(x.astype(np.float64))).astype(np.uint64)
    ids = (q % np.uint64(B)).astype(np.int64)
    _check(keys, B, gms.even_float_bucket(lower, float(inv)), ids, with_values=True)
    _check(keys, B, gms.even_float_bucket(lower, float(inv)), ids, with_values=False)
