"""Barriers written as inline PTX in the kernels, from their source - no GPU needed."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zap_b200", "csrc")


def test_named_barriers_do_not_assume_converged_warps():
    """bar.sync and barrier.sync.aligned are undefined when a warp's lanes reach them apart, and nothing in the source brings them
    together again after a branch: named barriers take the unaligned form. (The compiler orders __syncthreads itself.)"""
    aligned = re.compile(r'"[^"\n]*\b(bar(\.cta)?\.(sync|arrive|red)|barrier(\.cta)?\.(sync|arrive|red)\.aligned)\b')
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            found += [f"{os.path.basename(path)}:{k}" for k, line in enumerate(f, 1) if "asm" in line and aligned.search(line)]
    assert not found, found
