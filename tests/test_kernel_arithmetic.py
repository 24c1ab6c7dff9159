"""Arithmetic shortcuts of the kernels against the rules they stand for, over their whole domains, compiled for the host
(tests/host_emu/emu_arith.cu) - no GPU needed."""
import ctypes as C
import os
import shutil
import struct
import subprocess
from concurrent.futures import ThreadPoolExecutor

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "host_emu", "emu_arith.cu")
OUT = os.path.join(ROOT, "_build", "host_emu", "libztc_emu_arith.so")
CSRC = os.path.join(ROOT, "zap_b200", "csrc")
DEPS = [SRC] + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))]


@pytest.fixture(scope="module")
def emu():
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not available")
    if not os.path.exists(OUT) or os.path.getmtime(OUT) < max(os.path.getmtime(p) for p in DEPS):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.run(["nvcc", "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-fmad=false",
                        "-diag-suppress", "20091", "-Xcompiler", "-ffp-contract=off", "-Xcompiler", "-fPIC", "-shared",
                        "-o", OUT, SRC], check=True, capture_output=True)
    lib = C.CDLL(OUT)
    lib.emu_srgb_back_mismatches.argtypes = [C.c_uint64, C.c_uint64]
    lib.emu_srgb_back_mismatches.restype = C.c_uint64
    lib.emu_srgb_linear.restype = C.c_float
    lib.emu_bc4_distance_mismatches.restype = C.c_uint64
    return lib


def _bits(f):
    return struct.unpack("<I", struct.pack("<f", f))[0]


def test_srgb_one_word_search_equals_binary_search(emu):
    """Every float a sum of four linear values can be: 0, and from the least value above it to 4."""
    lo, hi, chunks = _bits(emu.emu_srgb_linear(1)), _bits(4.0) + 1, 64
    step = (hi - lo + chunks - 1) // chunks
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as ex:
        bad = sum(ex.map(lambda k: emu.emu_srgb_back_mismatches(lo + k * step, min(hi, lo + (k + 1) * step)), range(chunks)))
    assert bad + emu.emu_srgb_back_mismatches(0, 1) == 0


@pytest.mark.parametrize("ulps", [-4, 0, 4])
def test_bc4_distance_equals_palette_scan(emu, ulps):
    """Every endpoint pair and every level within the insets around it, at a reciprocal a few ulp off too."""
    assert emu.emu_bc4_distance_mismatches(ulps) == 0


def test_quant8_equals_three_candidate_search(emu):
    """The mode-6 endpoint quantiser for every float in [-512, 768] and both p-bits."""
    emu.emu_quant8_mismatches.argtypes = [C.c_uint64, C.c_uint64]
    emu.emu_quant8_mismatches.restype = C.c_uint64
    chunks = []
    for base, top in ((0, _bits(768.0) + 1), (0x80000000, 0x80000000 + _bits(512.0) + 1)):
        step = (top - base + 63) // 64
        chunks += [(base + k * step, min(top, base + (k + 1) * step)) for k in range(64)]
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as ex:
        assert sum(ex.map(lambda c: emu.emu_quant8_mismatches(*c), chunks)) == 0
