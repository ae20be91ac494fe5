"""Counts kept as rows (the one-call multisplit from 65 buckets and 512 tiles up): sizes around
the line and around whole ranges of tiles, the count matrix that the caller
finds afterwards, scratches with and without room for the rows, and every
operation built on such calls.  Whole numbers: every comparison is exact."""
import numpy as np
import pytest
import torch

import gpumultisplit_gb300 as gms
from gpu_util import host, identifiers, to_dev
from gpumultisplit_gb300 import datagen

pytestmark = pytest.mark.gpu

TILE = 4096


def _matrix_of(oracle_mod, keys, desc, tile):
    counts = oracle_mod.tile_counts(keys, desc, tile).astype(np.uint64)
    flat = counts.ravel()
    return (np.cumsum(flat) - flat).reshape(counts.shape).astype(np.uint32)


@pytest.mark.parametrize("B,kind", [(2, 4), (4, 0), (8, 0), (16, 2), (32, 3), (100, 1), (128, 0), (256, 0), (256, 3)])
@pytest.mark.parametrize("with_values", [False, True], ids=["keys", "pairs"])
def test_sizes_and_matrix(gms_lib, oracle_mod, B, kind, with_values):
    """609 to 1530 tiles: past the one-launch form, one and two tiles a range,
    ranges cut short, tile counts that are and are not multiples of eight."""
    o = oracle_mod
    ident, desc, keep = identifiers(o, kind, B)
    for n in (641 * TILE, 641 * TILE + 1, 760 * TILE, 761 * TILE + 17, 767 * TILE + 5, 1529 * TILE + 4095):
        keys = datagen.as_u32(datagen.uniform_u32(n, n % 1000 + B))
        vals = np.arange(n, dtype=np.uint32) if with_values else None
        dk = to_dev(keys)
        ok = torch.zeros_like(dk)
        dv = to_dev(vals) if with_values else None
        ov = torch.zeros_like(dk) if with_values else None
        rk, rv, roffs = o.multisplit(keys, desc, vals)
        want = _matrix_of(o, keys, desc, TILE)
        ctx = gms.multisplit_context(B)
        (gms.multisplit_allocate_key_value if with_values else gms.multisplit_allocate_key_only)(n, ctx)
        rows_bytes = 4 * (1 << (B - 1).bit_length()) * ctx.num_sub_prob if B > 64 else 0
        # the reported scratch, and the two smaller ones that were always taken
        for less in (0, rows_bytes, rows_bytes + (n + 255) // 256 * 256):
            ok.zero_()
            ctx.temp_storage_bytes = ctx.d_temp_storage.numel() - (less + 255) // 256 * 256
            ctx.d_temp_storage[256:].fill_(0x5A)
            if with_values:
                ov.zero_()
                offs = gms.multisplit_key_value(dk, dv, ok, ov, n, ctx, ident, True)
            else:
                offs = gms.multisplit_key_only(dk, ok, n, ctx, ident, True)
            assert gms.read_device_error(ctx) == 0
            assert offs == [int(x) for x in roffs], (n, less)
            np.testing.assert_array_equal(host(ok), rk, err_msg=f"keys, n={n}, less={less}")
            if with_values:
                np.testing.assert_array_equal(host(ov), rv, err_msg=f"values, n={n}, less={less}")
            m = ctx.d_histogram.cpu().numpy().view(np.uint32).reshape(B, ctx.num_sub_prob)
            np.testing.assert_array_equal(m, want, err_msg=f"matrix, n={n}, less={less}")
            assert bool((ctx.d_temp_storage[ctx.temp_storage_bytes:] == 0x5A).all()), "wrote past its scratch"


@pytest.mark.parametrize("n", [641 * TILE + 1, 5_000_011])
def test_operations_built_on_it(gms_lib, n):
    keys_t = datagen.uniform_u32(n, 5, device="cuda")
    keys = datagen.as_u32(keys_t)
    vals = datagen.index_values(n, "cuda")
    ko, vo = torch.empty_like(keys_t), torch.empty_like(vals)
    order = np.argsort(keys, kind="stable").astype(np.uint32)
    for bits in (4, 7, 8):
        ctx = gms.ms_sort_context()
        getattr(gms, f"multisplit_sort_{bits}bit_allocate_pairs")(n, ctx)
        getattr(gms, f"multisplit_sort_{bits}bit_pairs")(keys_t, ko, vals, vo, n, ctx)
        np.testing.assert_array_equal(host(vo), order)
    c = gms.compaction_context()
    gms.compaction_allocate_key_value(n, c)
    n0 = gms.compaction_key_value(keys_t, vals, ko, vo, n, c, gms.mask_bucket(8))
    odd = (keys & 8) != 0
    assert n0 == int((~odd).sum())
    np.testing.assert_array_equal(host(vo), np.argsort(odd, kind="stable").astype(np.uint32))
    for B in (257, 4096):
        ctx = gms.multisplit_context(B)
        gms.multisplit_allocate_key_value(n, ctx)
        offs = gms.multisplit_key_value(keys_t, vals, ko, vo, n, ctx, gms.delta_bucket(), True)
        ids = ((keys.astype(np.uint64) * np.uint64(B)) >> np.uint64(32)).astype(np.int64)
        np.testing.assert_array_equal(host(vo), np.argsort(ids, kind="stable").astype(np.uint32))
        cnt = np.bincount(ids, minlength=B)
        assert offs == [int(x) for x in np.cumsum(cnt) - cnt]


@pytest.mark.parametrize("widths", [(8, 0), (8, 4), (8, 8), (4, 8)])
def test_wide(gms_lib, widths):
    kb, vb = widths
    for n, B in ((641 * 4096 + 3, 256), (2_700_001, 8), (5_000_011, 100)):
        keys = datagen.uniform_u64(n, n, device="cuda") if kb == 8 else datagen.uniform_u32(n, n, device="cuda")
        h = datagen.as_u64(keys) if kb == 8 else datagen.as_u32(keys)
        vals = torch.arange(n, dtype=torch.int64 if vb == 8 else torch.int32, device="cuda") if vb else None
        ko, vo = torch.empty_like(keys), torch.empty_like(vals) if vb else None
        ctx = gms.multisplit_context(B)
        gms.multisplit_wide_allocate(n, ctx, kb, vb)
        offs = gms.multisplit_wide(keys, ko, n, ctx, gms.delta_bucket(), vals, vo, True)
        top = (h >> np.uint64(32)) if kb == 8 else h
        low = (h & np.uint64(0xFFFFFFFF)) if kb == 8 else np.zeros(n, np.uint64)
        top = top.astype(np.uint64)
        ids = ((top * np.uint64(B) + ((low * np.uint64(B)) >> np.uint64(32))) >> np.uint64(32)).astype(np.int64)
        order = np.argsort(ids, kind="stable")
        back = datagen.as_u64(ko) if kb == 8 else host(ko)
        np.testing.assert_array_equal(back, h[order])
        if vb:
            np.testing.assert_array_equal(vo.cpu().numpy(), order)
        cnt = np.bincount(ids, minlength=B)
        assert offs == [int(x) for x in np.cumsum(cnt) - cnt]


def test_repeated_calls_reset_the_scan(gms_lib):
    n, B = 700 * TILE, 256
    keys = datagen.uniform_u32(n, 3, device="cuda")
    out = torch.empty_like(keys)
    ctx = gms.multisplit_context(B)
    gms.multisplit_allocate_key_only(n, ctx)
    first = gms.multisplit_key_only(keys, out, n, ctx, gms.delta_bucket(), True)
    for _ in range(20):  # repeated calls reset ticket and status words
        assert gms.multisplit_key_only(keys, out, n, ctx, gms.delta_bucket(), True) == first
    assert gms.read_device_error(ctx) == 0
