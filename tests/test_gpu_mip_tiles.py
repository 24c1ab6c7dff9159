"""Mip launches whose CTAs take several tiles each, alone and with chains of different lengths in one launch, against the oracle."""
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import torch

import zap_b200

pytestmark = pytest.mark.gpu

CTAS_PER_SM, TILE = 4, 64  # resident CTAs of a mip launch, source texels a side of a tile


def _ctas():
    return CTAS_PER_SM * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("srgb", [0, 1])
def test_chain_of_several_tiles_per_cta(cuda_lib, oracle, srgb):
    """More than three tiles per CTA, ragged sides: both buffers of a CTA come round."""
    rows = int((3 * _ctas()) ** 0.5) + 1
    w, h = TILE * (rows + 2) - 7, TILE * rows - 9
    img = np.random.default_rng(srgb).integers(0, 256, (h, w, 4), dtype=np.uint8)
    img[h // 3:, : w // 2] = np.sort(img[h // 3:, : w // 2], axis=1)
    want = img
    for level in zap_b200.mip_chain_dev(torch.from_numpy(img).cuda(), srgb):
        want = oracle.mip_next(want, srgb)
        assert np.array_equal(level.cpu().numpy(), want), want.shape


def test_batch_of_long_and_short_chains(cuda_lib, oracle):
    """Chains of one to six levels in either mip launch (levels 1-6, then 7-12), more than two tiles per CTA in both: a tile of
    one level between two longer ones must not let the third take the first one's buffer too early."""
    shapes = [(512, 4, 0), (128, 4, 0), (256, 8, 0), (4, 130, 0), (512, 3, 0), (2, 2, 0), (3, 3, 0), (64, 64, 0), (16, 20, 2), (48, 33, 0)]
    long_shapes = [s for s in shapes if max(s[:2]) >= 128]  # one tile of the second launch each
    rng = np.random.default_rng(11)
    n = 2 * _ctas() + 200
    items = [shapes[i] for i in rng.integers(0, len(shapes), n)] + [long_shapes[i] for i in rng.integers(0, len(long_shapes), n)]
    items = [items[i] for i in rng.permutation(2 * n)]
    images = [rng.integers(0, 256, (h, w, 4), dtype=np.uint8) for w, h, _ in items]
    formats = [(zap_b200.BC1, zap_b200.BC4)[i] for i in rng.integers(0, 2, 2 * n)]
    srgb = [bool(i) for i in rng.integers(0, 2, 2 * n)]
    batch = zap_b200.Batch([torch.from_numpy(i).cuda() for i in images], formats, srgb=srgb, levels=[s[2] for s in items])

    def check(i):
        cur = images[i]
        for lv, view in enumerate(views[i]):
            if lv:
                cur = oracle.mip_next(cur, srgb[i] and formats[i] != zap_b200.BC4)
            if not np.array_equal(view, oracle.bc_encode(cur, formats[i])):
                return items[i], formats[i], lv
    for _ in range(2):
        batch.run()
        torch.cuda.synchronize()
        views = [[v.cpu().numpy() for v in batch.level_views(i)] for i in range(2 * n)]
        with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:  # the oracle's calls release the GIL
            bad = [b for b in pool.map(check, range(2 * n)) if b]
        assert not bad, (len(bad), bad[:8])
        for o in batch.outputs:
            o.fill_(0)
    batch.close()
