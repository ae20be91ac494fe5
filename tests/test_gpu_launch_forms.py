"""Which kernels a call launches: every form of the one-launch kernels (one block,
a cluster, a cooperative grid), the rows of counts and the three stages, each at
sizes picked for it.  The other tests compare outputs, which are the same when a
form silently gives way to another; here the call is captured and the kernels
read off the graph's nodes."""
import ctypes

import pytest
import torch

import gpumultisplit_gb300 as gms
from gpumultisplit_gb300 import datagen

pytestmark = pytest.mark.gpu

TILE = 4096


class _KernelNode(ctypes.Structure):  # CUDA_KERNEL_NODE_PARAMS (second version)
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("shared", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def launches(call):
    """(kernel, blocks, cooperative, cluster size) of every kernel that call(stream) launches."""
    cu = ctypes.CDLL("libcuda.so.1")

    def do(name, *args):
        st = getattr(cu, name)(*args)
        assert st == 0, (name, st)

    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    s, graph, count = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p(), ctypes.c_size_t()
    do("cuStreamBeginCapture_v2", s, 1)  # thread-local
    try:
        assert call(stream.cuda_stream) == 0
    finally:
        do("cuStreamEndCapture", s, ctypes.byref(graph))
    do("cuGraphGetNodes", graph, None, ctypes.byref(count))
    nodes = (ctypes.c_void_p * count.value)()
    do("cuGraphGetNodes", graph, nodes, ctypes.byref(count))
    out = []
    for node in nodes:
        node, kind, p, name = ctypes.c_void_p(node), ctypes.c_int(), _KernelNode(), ctypes.c_char_p()
        do("cuGraphNodeGetType", node, ctypes.byref(kind))
        if kind.value != 0:  # a kernel
            continue
        do("cuGraphKernelNodeGetParams_v2", node, ctypes.byref(p))
        if p.kern:
            do("cuKernelGetName", ctypes.byref(name), ctypes.c_void_p(p.kern))
        else:
            do("cuFuncGetName", ctypes.byref(name), ctypes.c_void_p(p.func))
        value = (ctypes.c_uint * 16)()  # a launch attribute's value: 64 bytes
        do("cuGraphKernelNodeGetAttribute", node, 2, value)
        cooperative = value[0]
        value = (ctypes.c_uint * 16)()
        do("cuGraphKernelNodeGetAttribute", node, 4, value)
        known = ["fused_sort_kernel", "fused_kernel", "scan_rows_kernel", "prescan64_kernel", "prescan_kernel",
                 "postscan_persistent_kernel", "postscan_kernel", "scan_kernel"]
        mangled = name.value.decode()
        short = next((k for k in known if f"{len(k)}{k}" in mangled), mangled)
        out.append((short, p.grid[0], bool(cooperative), max(value[0], 1)))
    do("cuGraphDestroy", graph)
    return out


def _resident(per_sm):
    return per_sm * torch.cuda.get_device_properties(0).multi_processor_count


def _split(lib, n, B, pairs, ident, less=0):
    k = datagen.uniform_u32(n, 1, device="cuda")
    v, ko, vo = (torch.empty_like(k) for _ in range(3))
    ctx = gms.multisplit_context(B)
    (gms.multisplit_allocate_key_value if pairs else gms.multisplit_allocate_key_only)(n, ctx)
    keep = datagen.range_splitters(B, 5, device="cuda")
    d = (gms.range_bucket(keep) if ident == "range" else gms.delta_bucket()).desc(B)
    scratch, nbytes = ctx.d_temp_storage, ctx.temp_storage_bytes - less

    def call(s):
        if pairs:
            return lib.gms_multisplit_key_value(k.data_ptr(), v.data_ptr(), ko.data_ptr(), vo.data_ptr(), n,
                                                ctypes.byref(d), scratch.data_ptr(), nbytes, None, s)
        return lib.gms_multisplit_key_only(k.data_ptr(), ko.data_ptr(), n, ctypes.byref(d), scratch.data_ptr(),
                                           nbytes, None, s)

    call.keep = (k, v, ko, vo, keep)
    assert call(torch.cuda.current_stream().cuda_stream) == 0
    return launches(call)


@pytest.mark.parametrize("ident", ["delta", "range"])
@pytest.mark.parametrize("pairs", [False, True], ids=["keys", "pairs"])
@pytest.mark.parametrize("B", [8, 256])
def test_multisplit(gms_lib, B, pairs, ident):
    one = lambda tiles, less=0: _split(gms_lib, tiles * TILE - 7, B, pairs, ident, less)  # noqa: E731
    assert one(1) == [("fused_kernel", 1, False, 1)]
    for tiles, blocks in ((2, 2), (3, 4), (9, 16), (16, 16)):
        assert one(tiles) == [("fused_kernel", blocks, False, blocks)]
        # no room for the counts: they stay in the cluster's shared memory
        assert one(tiles, (tiles * TILE - 7 + 255) // 256 * 256) == [("fused_kernel", blocks, False, blocks)]
    # Blocks on an SM at once: four, but three of the 256-bucket range pairs', whose
    # tile, count table and splitters take 67 KB of its 228.
    resident = _resident(3 if (B, pairs, ident) == (256, True, "range") else 4)
    most = min(448 if pairs and ident == "delta" else 640, _resident(4))
    for tiles in (17, 33, 200, min(most, resident), most):
        got = one(tiles)
        if tiles <= resident:
            assert got == [("fused_kernel", tiles, True, 1)]
        else:
            assert [x[0] for x in got] == ["prescan_kernel", "scan_rows_kernel", "postscan_kernel"]
    names = [x[0] for x in one(641)]
    assert names == ["prescan_kernel", "scan_rows_kernel" if B == 256 else "scan_kernel", "postscan_kernel"]


def test_stages_with_little_scratch(gms_lib):
    """Beyond a cluster the counts need room: without it, the three stages over the matrix."""
    n = 40 * TILE
    assert [x[0] for x in _split(gms_lib, n, 256, False, "delta", n)] == ["prescan_kernel", "scan_kernel", "postscan_kernel"]
    assert [x[0] for x in _split(gms_lib, n, 256, False, "range", n)] == \
        ["prescan_kernel", "scan_kernel", "postscan_persistent_kernel"]
    n = 700 * TILE
    less = 256 * 700 * 4
    assert [x[0] for x in _split(gms_lib, n, 256, True, "delta", less + n)] == \
        ["prescan_kernel", "scan_kernel", "postscan_kernel"]


@pytest.mark.parametrize("pairs", [False, True], ids=["keys", "pairs"])
def test_sorts(gms_lib, pairs):
    def sort(n, bits, method=None):
        k = datagen.uniform_u32(n, 2, device="cuda")
        v, ko, vo = (torch.empty_like(k) for _ in range(3))
        nbytes = ctypes.c_size_t()
        assert gms_lib.gms_sort_scratch_bytes(n, bits, int(pairs), ctypes.byref(nbytes)) == 0
        scratch = torch.empty(nbytes.value, dtype=torch.uint8, device="cuda")

        def call(s):
            if pairs:
                return gms_lib.gms_sort_key_value(k.data_ptr(), ko.data_ptr(), v.data_ptr(), vo.data_ptr(), n, bits,
                                                  scratch.data_ptr(), nbytes.value, s)
            return gms_lib.gms_sort_key_only(k.data_ptr(), ko.data_ptr(), n, bits, scratch.data_ptr(), nbytes.value, s)

        assert call(torch.cuda.current_stream().cuda_stream) == 0
        return launches(call)

    assert sort(1000, 8) == [("fused_sort_kernel", 1, False, 1)]
    assert sort(2048, 7) == [("fused_sort_kernel", 1, False, 1)]
    assert sort(10000, 8) == [("fused_sort_kernel", 16, False, 16)]
    assert sort(30000, 4) == [("fused_sort_kernel", 16, False, 16)]
    assert sort(65536, 8) == [("fused_sort_kernel", 16, False, 16)]
    assert sort(300000, 8) == [("fused_sort_kernel", (300000 + 2047) // 2048, True, 1)]
    tiles = min(608, _resident(4))
    assert sort(tiles * TILE, 8) == [("fused_sort_kernel", tiles, True, 1)]
    assert [x[0] for x in sort(3000000, 8)] == ["prescan_kernel", "scan_rows_kernel", "postscan_kernel"] * 4


def test_wide_and_many_buckets(gms_lib):
    def wide(n, B):
        k = datagen.uniform_u64(n, 3, device="cuda")
        ko = torch.empty_like(k)
        ctx = gms.multisplit_context(B)
        gms.multisplit_wide_allocate(n, ctx, 8, 0)
        d = gms.delta_bucket().desc64(B)

        def call(s):
            return gms_lib.gms_multisplit_wide(k.data_ptr(), None, ko.data_ptr(), None, n, 8, 0, ctypes.byref(d),
                                               ctx.d_temp_storage.data_ptr(), ctx.temp_storage_bytes, None, s)

        assert call(torch.cuda.current_stream().cuda_stream) == 0
        return launches(call)

    assert wide(1000, 64) == [("fused_kernel", 1, False, 1)]
    assert wide(20000, 256)[0][0] == "fused_kernel" and wide(20000, 256)[0][3] > 1
    assert wide(300000, 256)[0][:1] + wide(300000, 256)[0][2:] == ("fused_kernel", True, 1)
    assert [x[0] for x in wide(4000000, 256)] == ["prescan64_kernel", "scan_rows_kernel", "postscan_kernel"]
    # above 256 buckets: two digit passes, each one launch
    assert [x[0] for x in _split(gms_lib, 100 * TILE, 4096, True, "range")] == ["fused_kernel"] * 2
    assert [x[0] for x in _split(gms_lib, 900 * TILE, 65536, True, "delta")] == \
        ["prescan_kernel", "scan_rows_kernel", "postscan_kernel"] * 2
