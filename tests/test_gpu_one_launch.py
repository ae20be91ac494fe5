"""Multisplits small enough to run as one launch: the sizes where the launch
form changes (one tile, one thread-block cluster, a cooperative grid, one
barrier or two, the largest it takes and the next), against the oracle.
Whole numbers: every comparison is exact."""
import ctypes

import numpy as np
import pytest
import torch

import gpumultisplit_gb300 as gms
from gpu_util import host, identifiers, run_multisplit, to_dev
from gpumultisplit_gb300 import datagen

pytestmark = pytest.mark.gpu

TILE = 4096
# tiles: 1 | cluster 2..16 | grid; 8192 counts are the most one barrier adds up
# (32 tiles at 256 buckets, 256 at 32); pairs with a cheap identifier stop at
# 448 tiles, the others at what is resident (608 on 152 SMs) or 640.
SIZES = [1, 31, TILE - 1, TILE, TILE + 1, 2 * TILE + 3, 8 * TILE, 8 * TILE + 1, 16 * TILE, 16 * TILE + 1,
         32 * TILE, 32 * TILE + 5, 64 * TILE + 2, 256 * TILE, 257 * TILE, 448 * TILE, 448 * TILE + 1, 608 * TILE,
         608 * TILE + 1]


def _matrix_of(oracle_mod, keys, desc, tile):
    """The scanned count matrix: exclusive scan of the per-tile counts, bucket-major."""
    counts = oracle_mod.tile_counts(keys, desc, tile).astype(np.uint64)
    flat = counts.ravel()
    return (np.cumsum(flat) - flat).reshape(counts.shape).astype(np.uint32)


@pytest.mark.parametrize("B,kind", [(2, 4), (8, 0), (32, 0), (100, 1), (128, 2), (256, 0), (256, 3), (32, 3), (7, 5)])
@pytest.mark.parametrize("with_values", [False, True], ids=["keys", "pairs"])
def test_sizes_around_each_form(gms_lib, oracle_mod, B, kind, with_values):
    o = oracle_mod
    ident, desc, keep = identifiers(o, kind, B)
    for n in SIZES:
        keys = datagen.as_u32(datagen.uniform_u32(n, n + B))
        vals = np.arange(n, dtype=np.uint32) if with_values else None
        dk, ok = to_dev(keys), to_dev(np.zeros(n, np.uint32))
        dv, ov = (to_dev(vals), to_dev(np.zeros(n, np.uint32))) if with_values else (None, None)
        ctx = gms.multisplit_context(B)
        if with_values:
            gms.multisplit_allocate_key_value(n, ctx)
            offs = gms.multisplit_key_value(dk, dv, ok, ov, n, ctx, ident, True)
        else:
            gms.multisplit_allocate_key_only(n, ctx)
            offs = gms.multisplit_key_only(dk, ok, n, ctx, ident, True)
        assert gms.read_device_error(ctx) == 0
        rk, rv, roffs = o.multisplit(keys, desc, vals)
        np.testing.assert_array_equal(host(ok), rk, err_msg=f"keys, n={n}")
        if with_values:
            np.testing.assert_array_equal(host(ov), rv, err_msg=f"values, n={n}")
        assert offs == [int(x) for x in roffs], n
        m = ctx.d_histogram.cpu().numpy().view(np.uint32).reshape(B, ctx.num_sub_prob)
        np.testing.assert_array_equal(m, _matrix_of(o, keys, desc, ctx.size_sub_prob), err_msg=f"matrix, n={n}")


@pytest.mark.parametrize("n", [3 * TILE + 7, 20 * TILE + 1, 300 * TILE + 9])
@pytest.mark.parametrize("B", [8, 256])
@pytest.mark.parametrize("misalign", [1, 2])
def test_arrays_off_a_16_byte_boundary(gms_lib, oracle_mod, n, B, misalign):
    o = oracle_mod
    ident, desc, _ = identifiers(o, o.DELTA, B)
    keys = datagen.as_u32(datagen.uniform_u32(n, 5))
    vals = np.arange(n, dtype=np.uint32)
    gk, gv, offs, err = run_multisplit(keys, B, ident, vals, misalign=misalign)
    rk, rv, roffs = o.multisplit(keys, desc, vals)
    assert err == 0 and offs == [int(x) for x in roffs]
    np.testing.assert_array_equal(gk, rk)
    np.testing.assert_array_equal(gv, rv)


@pytest.mark.parametrize("n", [5 * TILE, 100 * TILE + 3])
def test_skewed_keys(gms_lib, oracle_mod, n):
    """All keys in one bucket, and in two far apart: counts of a whole tile."""
    o = oracle_mod
    ident, desc, _ = identifiers(o, o.DELTA, 256)
    for keys in (np.full(n, 0x7F001234, np.uint32), np.where(np.arange(n) % 3 == 0, 0, 0xFFFFFFFF).astype(np.uint32)):
        vals = np.arange(n, dtype=np.uint32)
        gk, gv, offs, err = run_multisplit(keys, 256, ident, vals)
        rk, rv, roffs = o.multisplit(keys, desc, vals)
        assert err == 0 and offs == [int(x) for x in roffs]
        np.testing.assert_array_equal(gk, rk)
        np.testing.assert_array_equal(gv, rv)


@pytest.mark.parametrize("n", [1, TILE + 1, 16 * TILE, 100 * TILE + 1])
@pytest.mark.parametrize("kind", [0, 3], ids=["delta", "range"])
def test_smallest_accepted_scratch(gms_lib, oracle_mod, n, kind):
    """A scratch without the byte per key is taken as before, with the same output."""
    o = oracle_mod
    B = 256
    ident, desc, keep = identifiers(o, kind, B)
    keys = datagen.as_u32(datagen.uniform_u32(n, 11))
    dk, ok = to_dev(keys), to_dev(np.zeros(n, np.uint32))
    ctx = gms.multisplit_context(B)
    gms.multisplit_allocate_key_only(n, ctx)
    smallest = ctx.temp_storage_bytes - (n + 255) // 256 * 256
    d = ident.desc(B)
    lib, s = gms_lib, torch.cuda.current_stream().cuda_stream
    for nbytes, want in ((smallest - 256, 3), (smallest, 0), (smallest + 256, 0)):
        st = lib.gms_multisplit_key_only(dk.data_ptr(), ok.data_ptr(), n, ctypes.byref(d),
                                         ctx.d_temp_storage.data_ptr(), nbytes, None, s)
        assert st == want, (nbytes, st)
        if want == 0:
            np.testing.assert_array_equal(host(ok), o.multisplit(keys, desc)[0])
            ok.zero_()


def test_two_streams_and_a_captured_graph(gms_lib, oracle_mod):
    """Calls of every form on two streams at once, each with its scratch, and
    the same calls replayed from one CUDA graph on new keys."""
    o = oracle_mod
    B = 64
    ident, desc, _ = identifiers(o, o.DELTA, B)
    jobs = []
    for i, n in enumerate((TILE, 9 * TILE + 1, 40 * TILE + 3, 300 * TILE)):
        keys = datagen.as_u32(datagen.uniform_u32(n, 50 + i))
        vals = np.arange(n, dtype=np.uint32)
        ctx = gms.multisplit_context(B)
        gms.multisplit_allocate_key_value(n, ctx)
        dk, dv = to_dev(keys), to_dev(vals)
        jobs.append((n, ctx, keys, vals, dk, dv, torch.zeros_like(dk), torch.zeros_like(dv)))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(20):
        for i, (n, ctx, _, _, dk, dv, ok, ov) in enumerate(jobs):
            with torch.cuda.stream(streams[i % 2]):
                gms.multisplit_key_value(dk, dv, ok, ov, n, ctx, ident)
    torch.cuda.synchronize()

    def check():
        for n, ctx, keys, vals, dk, dv, ok, ov in jobs:
            rk, rv, _ = o.multisplit(host(dk), desc, vals)
            np.testing.assert_array_equal(host(ok), rk)
            np.testing.assert_array_equal(host(ov), rv)
            assert gms.read_device_error(ctx) == 0

    check()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=streams[0]):
        for n, ctx, _, _, dk, dv, ok, ov in jobs:
            gms.multisplit_key_value(dk, dv, ok, ov, n, ctx, ident)
    for rep in range(3):
        for n, _, _, _, dk, _, ok, ov in jobs:
            dk.copy_(datagen.uniform_u32(n, 900 + rep, device="cuda"))
            ok.zero_(), ov.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        check()


# ---------------------------------------------------------------- sorts in one launch
# keys per block 1024 / 2048 / 4096: one block, one cluster of 16, a grid; the
# largest size and the next one, and one that is not taken.
SORT_SIZES = [1, 2, 1023, 1024, 1025, 2048, 2049, 4097, 16384, 16385, 32768, 32769, 65536, 65537, 100003, 400000,
              400001, 1000003, 2490368, 2490369]


def _sort_call(gms_lib, bits, kin, kout, vin, vout, n, scratch, nbytes):
    s = torch.cuda.current_stream().cuda_stream
    if vin is None:
        return gms_lib.gms_sort_key_only(kin.data_ptr(), kout.data_ptr(), n, bits, scratch.data_ptr(), nbytes, s)
    return gms_lib.gms_sort_key_value(kin.data_ptr(), kout.data_ptr(), vin.data_ptr(), vout.data_ptr(), n, bits,
                                      scratch.data_ptr(), nbytes, s)


@pytest.mark.parametrize("bits", [4, 7, 8])
@pytest.mark.parametrize("with_values", [False, True], ids=["keys", "pairs"])
def test_sort_sizes(gms_lib, bits, with_values):
    """Every form, against numpy's stable argsort; the reported scratch, and one
    without the count rows at its end, which must still be taken."""
    for n in SORT_SIZES:
        keys = datagen.as_u32(datagen.and4_u32(n, n + bits) if n % 2 else datagen.uniform_u32(n, n))
        order = np.argsort(keys, kind="stable")
        sb = ctypes.c_size_t()
        assert gms_lib.gms_sort_scratch_bytes(n, bits, int(with_values), ctypes.byref(sb)) == 0
        tile = 1024 if n <= 16384 else 2048 if n <= 400000 else 4096
        rows = ((n + tile - 1) // tile * 1024 + 1024 + 255) // 256 * 256 if n <= 2500000 else 0
        for nbytes in {sb.value, sb.value - rows}:
            kin, kout = to_dev(keys), to_dev(np.zeros(n, np.uint32))
            vin = to_dev(np.arange(n, dtype=np.uint32)) if with_values else None
            vout = torch.zeros_like(vin) if with_values else None
            scratch = torch.full((sb.value,), 0x5A, dtype=torch.uint8, device="cuda")  # nothing in it is assumed
            scratch[nbytes:].fill_(0x33)
            assert _sort_call(gms_lib, bits, kin, kout, vin, vout, n, scratch, nbytes) == 0
            np.testing.assert_array_equal(host(kout), keys[order], err_msg=f"keys, n={n}, scratch={nbytes}")
            if with_values:
                np.testing.assert_array_equal(host(vout), order.astype(np.uint32), err_msg=f"values, n={n}")
            assert bool((scratch[nbytes:] == 0x33).all()), "wrote past the scratch it was given"
            np.testing.assert_array_equal(host(kin), keys, err_msg="the input changed")


@pytest.mark.parametrize("n", [700, 5000, 50001, 300007, 1500001])
def test_sort_bits_ranges(gms_lib, n):
    """Key bits [begin, end) whose last digit is narrow, in one launch."""
    keys_t = datagen.uniform_u32(n, n, device="cuda")
    keys = datagen.as_u32(keys_t)
    for begin, end, digit in ((3, 17, 5), (20, 21, 6), (0, 9, 8), (8, 32, 8), (31, 32, 4)):
        ctx = gms.ms_sort_context()
        gms.multisplit_sort_bits_allocate(n, ctx, begin, end, digit, pairs=True)
        vin = datagen.index_values(n, "cuda")
        ko, vo = torch.empty_like(keys_t), torch.empty_like(vin)
        gms.multisplit_sort_bits_pairs(keys_t, ko, vin, vo, n, ctx)
        field = (keys >> np.uint32(begin)) & np.uint32((1 << (end - begin)) - 1)
        order = np.argsort(field, kind="stable")
        np.testing.assert_array_equal(host(vo), order.astype(np.uint32), err_msg=f"{begin, end, digit}")
        np.testing.assert_array_equal(host(ko), keys[order])


@pytest.mark.parametrize("widths", [(8, 0), (8, 4), (8, 8), (4, 8)])
def test_wide_sizes(gms_lib, widths):
    """Multisplits and sorts of 64-bit elements around each form's limits."""
    kb, vb = widths
    for n in (1, 1024, 1025, 2049, 3072, 3073, 16384, 16385, 32769, 16 * 3072 + 1, 65537, 300001, 456 * 3072,
              456 * 3072 + 1, 1999999, 2000001):
        keys = datagen.uniform_u64(n, n, device="cuda") if kb == 8 else datagen.uniform_u32(n, n, device="cuda")
        h = datagen.as_u64(keys) if kb == 8 else datagen.as_u32(keys)
        vals = torch.arange(n, dtype=torch.int64 if vb == 8 else torch.int32, device="cuda") if vb else None
        ko, vo = torch.empty_like(keys), torch.empty_like(vals) if vb else None
        ctx = gms.ms_sort_context()
        gms.multisplit_sort_wide_allocate(n, ctx, kb, vb)
        gms.multisplit_sort_wide(keys, ko, n, ctx, vals, vo)
        order = np.argsort(h, kind="stable")
        back = datagen.as_u64(ko) if kb == 8 else host(ko)
        np.testing.assert_array_equal(back, h[order], err_msg=f"sorted keys, n={n}")
        if vb:
            np.testing.assert_array_equal(vo.cpu().numpy(), order, err_msg=f"sorted values, n={n}")
        for B in (8, 256):
            ms = gms.multisplit_context(B)
            gms.multisplit_wide_allocate(n, ms, kb, vb)
            offs = gms.multisplit_wide(keys, ko, n, ms, gms.delta_bucket(), vals, vo, True)
            ids = (h >> h.dtype.type(8 * kb - (B.bit_length() - 1))).astype(np.int64)
            order = np.argsort(ids, kind="stable")
            back = datagen.as_u64(ko) if kb == 8 else host(ko)
            np.testing.assert_array_equal(back, h[order], err_msg=f"keys, n={n}, B={B}")
            if vb:
                np.testing.assert_array_equal(vo.cpu().numpy(), order, err_msg=f"values, n={n}, B={B}")
            c = np.bincount(ids, minlength=B)
            assert offs == [int(x) for x in np.cumsum(c) - c]


def test_sort_in_place_keeps_its_route(gms_lib):
    """An even number of passes takes kin == kout (8-bit digits), as before."""
    for n in (1000, 30000, 200001):
        keys = datagen.as_u32(datagen.uniform_u32(n, 4))
        sb = ctypes.c_size_t()
        assert gms_lib.gms_sort_scratch_bytes(n, 8, 0, ctypes.byref(sb)) == 0
        k = to_dev(keys)
        scratch = torch.empty(sb.value, dtype=torch.uint8, device="cuda")
        assert _sort_call(gms_lib, 8, k, k, None, None, n, scratch, sb.value) == 0
        np.testing.assert_array_equal(host(k), np.sort(keys))
        # an odd number refuses it, as before
        assert gms_lib.gms_sort_scratch_bytes(n, 7, 0, ctypes.byref(sb)) == 0
        scratch = torch.empty(sb.value, dtype=torch.uint8, device="cuda")
        assert _sort_call(gms_lib, 7, k, k, None, None, n, scratch, sb.value) == 1
