"""zap_tex_cuda_reserve sets what a context's scratch pool keeps: more, less, or nothing."""
import ctypes as C

import numpy as np
import pytest
import torch

import zap_b200

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture
def ctx(cuda_lib):
    lib, c = zap_b200.load(), C.c_void_p()
    zap_b200.bc_encode_dev(torch.zeros(8, 8, 4, dtype=torch.uint8, device="cuda"), zap_b200.BC7)  # first-call set-up is behind us
    zap_b200.check(lib.zap_tex_cuda_create(0, C.byref(c)), "create")
    yield c
    lib.zap_tex_cuda_destroy(c)


@pytest.mark.parametrize("sizes", [(40, 0), (128, 0), (256, 96, 0), (8, 256, 0), (300, 7, 0)])
def test_reserve_raises_and_lowers_what_is_kept(ctx, sizes):
    """Free device memory follows the figure, up to the step of 32 MB in which a pool holds it (and 4 MB for what else moves)."""
    base = _free()
    for mb in sizes:
        zap_b200.check(zap_b200.load().zap_tex_cuda_reserve(ctx, mb * MB), "reserve")
        held = base - _free()
        assert mb * MB <= held <= ((mb + 31) // 32 * 32 + 4) * MB, (mb, held / MB)


def test_reserve_zero_gives_back_what_calls_used(ctx, oracle):
    """After a call that left its scratch in the pool; the next call works as before."""
    img = torch.randint(0, 256, (4096, 8192, 4), dtype=torch.uint8, device="cuda")  # 16 MB of scratch
    out = torch.empty(zap_b200.bc_size(8192, 4096, zap_b200.BC7), dtype=torch.uint8, device="cuda")
    base = _free()
    zap_b200.bc_encode_dev(img, zap_b200.BC7, out=out, ctx=ctx)
    assert base - _free() >= 16 * MB  # kept
    zap_b200.check(zap_b200.load().zap_tex_cuda_reserve(ctx, 0), "reserve")
    assert base - _free() <= 4 * MB
    small = img[:60, :100]
    got = zap_b200.bc_encode_dev(small, zap_b200.BC7, ctx=ctx).cpu().numpy()
    assert np.array_equal(got, oracle.bc_encode(np.ascontiguousarray(small.cpu().numpy()), zap_b200.BC7))


@pytest.mark.parametrize("huge", [1 << 62, (1 << 64) - 1])
def test_reserve_that_fails_changes_nothing(ctx, huge):
    """A figure beyond the device's memory: what is held stays, and so does the figure that was in force."""
    img = torch.randint(0, 256, (4096, 8192, 4), dtype=torch.uint8, device="cuda")  # a rate-distortion call uses 128 MB of scratch
    out = torch.empty(zap_b200.bc_size(8192, 4096, zap_b200.BC7), dtype=torch.uint8, device="cuda")
    zap_b200.bc_encode_dev(img, zap_b200.BC7, out=out)
    base = _free()
    zap_b200.check(zap_b200.load().zap_tex_cuda_reserve(ctx, 64 * MB), "reserve")
    assert zap_b200.load().zap_tex_cuda_reserve(ctx, huge) != 0
    assert base - _free() >= 64 * MB
    zap_b200.bc_encode_rdo_dev(img, zap_b200.BC7, 30.0, band_rows=1, out=out, ctx=ctx)
    assert base - _free() <= (64 + 4) * MB


def test_reserve_without_memory_keeps_the_figure(ctx):
    """An allocation that fails on the way, made on the host: the figure in force before stays."""
    lib = zap_b200.load()
    zap_b200.check(lib.zap_tex_cuda_reserve(ctx, 0), "reserve")
    base = _free()
    lib.zap_tex_cuda_debug_fail_allocations(0, 1)
    try:
        assert lib.zap_tex_cuda_reserve(ctx, 256 * MB) == -4
    finally:
        lib.zap_tex_cuda_debug_fail_allocations(0, 0)
    img = torch.randint(0, 256, (4096, 8192, 4), dtype=torch.uint8, device="cuda")
    out = torch.empty(zap_b200.bc_size(8192, 4096, zap_b200.BC7), dtype=torch.uint8, device="cuda")
    used = base - _free()
    zap_b200.bc_encode_dev(img, zap_b200.BC7, out=out, ctx=ctx)  # 16 MB of scratch
    assert base - _free() - used <= 4 * MB
