"""The prescan's ranges of tiles: on the host, that they cover every tile and are
whole groups only where that costs little; on the GPU, the counts that the
stage entry point writes, for tile counts whose ranges start and end inside a
group of the matrix and for ranges of whole groups.  Whole numbers: exact."""
import ctypes
import subprocess
from pathlib import Path

import pytest

from gpumultisplit_gb300 import build as gbuild

ROOT = Path(__file__).resolve().parent.parent
TILE = 4096


def test_ranges_on_the_host(tmp_path):
    exe = tmp_path / "ranges_test"
    subprocess.run([gbuild.nvcc_path(), *gbuild.ARCH_FLAGS, "-std=c++17", "-I", str(ROOT / "include"), "-I",
                    str(ROOT / "gpumultisplit_gb300" / "csrc"), str(ROOT / "tests" / "cpp" / "ranges_test.cu"), "-o",
                    str(exe)], check=True, stdout=subprocess.DEVNULL, stderr=subprocess.DEVNULL)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


# With 608 to 1216 blocks: one tile a block, 2 to 12, about 17, and (last) 44 to 88 of them.
@pytest.mark.gpu
@pytest.mark.parametrize("tiles", [1, 7, 609, 1217, 8191, 8193, 13007, 46387])
@pytest.mark.parametrize("B", [2, 16, 64, 128, 256])
def test_counts_of_the_stage_call(gms_lib, tiles, B):
    import torch

    import gpumultisplit_gb300 as gms
    from gpumultisplit_gb300 import datagen

    n = tiles * TILE - 5
    keys = datagen.uniform_u32(n, tiles + B, device="cuda")
    ctx = gms.multisplit_context(B)
    gms.multisplit_allocate_key_only(n, ctx)
    ctx.d_temp_storage[256:].fill_(0x5A)
    s = torch.cuda.current_stream().cuda_stream
    d = gms.delta_bucket().desc(B)
    assert gms_lib.gms_multisplit_prescan(keys.data_ptr(), n, ctypes.byref(d), 0, ctx.d_temp_storage.data_ptr(),
                                          ctx.temp_storage_bytes, s) == 0
    bits = B.bit_length() - 1
    ids = (keys >> (32 - bits)) & (B - 1)
    tile = torch.arange(n, device="cuda", dtype=torch.int32) // TILE
    want = torch.bincount(ids * tiles + tile, minlength=B * tiles)
    assert torch.equal(ctx.d_histogram.to(torch.int64), want)
