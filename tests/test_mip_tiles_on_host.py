"""The order of the mip generator's tiles within a CTA, on the host (tests/host_emu/emu_mip.cpp) - no GPU needed.

A CTA of a batch takes tiles of chains of different lengths one after another, and one warp finishes a tile's small levels while
the others go on to the next. Each run keeps one warp back as far as the kernel's barriers let it fall behind; every
level must still be the box filter's bytes.
"""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "host_emu", "emu_mip.cpp")
CSRC = os.path.join(ROOT, "zap_b200", "csrc")
BUILD = os.path.join(ROOT, "_build", "host_emu")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

FULL, TWO = 6, 2  # levels of a launch: all six, and a chain cut short by the caller


@pytest.fixture(scope="module")
def emu():
    if shutil.which("g++") is None or not os.path.isdir(os.path.join(CUDA, "include")):
        pytest.skip("g++ and the CUDA headers needed")
    os.makedirs(BUILD, exist_ok=True)
    with open(os.path.join(CSRC, "mip.cu")) as f:
        text = f.read()
    part = os.path.join(BUILD, "mip_tiles.inc")
    with open(part, "w") as f:  # what stands before the first kernel
        f.write(text[:text.index("template <bool SRGB>\n__global__")] + "}  // namespace ztc\n")
    out = os.path.join(BUILD, "libztc_emu_mip.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fno-strict-aliasing", "-w", "-fPIC", "-shared", "-I", CSRC, "-I", os.path.join(CUDA, "include"),
                    f'-DEMU_MIP_SOURCE="{part}"', "-o", out, SRC], check=True)
    return C.CDLL(out)


def _next(img):
    h, w = img.shape[:2]
    nh, nw = max(1, h // 2), max(1, w // 2)
    y, x = np.arange(nh) * 2, np.arange(nw) * 2
    y1, x1 = np.minimum(y + 1, h - 1), np.minimum(x + 1, w - 1)
    v = img.astype(np.uint32)
    return ((v[y][:, x] + v[y][:, x1] + v[y1][:, x] + v[y1][:, x1] + 2) >> 2).astype(np.uint8)


def _run(emu, sizes, slow, seed):
    """sizes: (w, h, levels) per chain; levels are cut to those the size has."""
    rng = np.random.default_rng(seed)
    src, dst, want, levels = [], [], [], []
    for w, h, n in sizes:
        img = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
        n = min(n, max(w, h).bit_length() - 1)
        src.append(img)
        levels.append(n)
        for _ in range(n):
            img = _next(img)
            want.append(img)
            dst.append(np.zeros(img.shape, np.uint8))
        dst += [np.zeros(1, np.uint8)] * (6 - n)
        want += [np.zeros(1, np.uint8)] * (6 - n)
    n = len(sizes)
    ptr = lambda arrays: (C.c_void_p * len(arrays))(*[a.ctypes.data for a in arrays])
    ints = lambda values: (C.c_int * n)(*values)
    st = emu.emu_mip_chains(n, ptr(src), ints([a.shape[1] for a in src]), ints([a.shape[0] for a in src]), ints(levels), ptr(dst), slow)
    assert st == 0
    for k, (d, e) in enumerate(zip(dst, want)):
        assert np.array_equal(d, e), (sizes[k // 6], k % 6 + 1, slow)


@pytest.mark.parametrize("slow", range(8))
@pytest.mark.parametrize("between", [(2, 2, FULL), (3, 3, FULL), (16, 16, TWO), (1, 2, FULL), (64, 64, 1), (5, 4, FULL)])
def test_short_chains_between_long_ones(emu, between, slow):
    """One, two and three short chains between long ones, so that each of the two buffers comes round at every distance."""
    sizes = []
    for k in range(3):
        sizes += [(64, 64, FULL)] + [between] * (k + 1) + [(48, 64, FULL), (64, 33, FULL)]
    _run(emu, sizes, slow, slow)


@pytest.mark.parametrize("slow", range(8))
def test_mixed_chains(emu, slow):
    rng = np.random.default_rng(5 + slow)
    kinds = [(64, 64, FULL), (130, 70, FULL), (2, 2, FULL), (3, 2, FULL), (8, 8, FULL), (4, 1, FULL), (64, 64, TWO), (100, 90, 3)]
    _run(emu, [kinds[i] for i in rng.integers(0, len(kinds), 40)], slow, slow)
