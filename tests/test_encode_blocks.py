"""The device image encoder over blocks of images (four cells and several
images a thread) against the oracle's: frame sizes that are no
multiple of four, frames off 4-byte alignment, image counts around a thread's
share, cells outside the images kept (tolerance: exact)."""
import numpy as np
import pytest

import oracle
from bismit_b200 import cortex, encode as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dims,pad,offset", [(1, (13, 19), 0, 0), (33, (13, 19), 3, 1), (700, (64, 64), 0, 0),
                                               (129, (30, 50), 0, 2), (5, (1, 3), 1, 0), (64, (128, 128), 4, 0)])
def test_blocks_match_oracle(n, dims, pad, offset):
    import torch
    ctx = cortex._Ctx(0)
    rng = np.random.default_rng([n, dims[0]])
    ys, xs = 28, 20
    imgs = rng.integers(0, 256, (n, ys, xs), dtype=np.uint8)
    stride = dims[0] * dims[1] + pad
    frames = rng.integers(0, 256, n * stride + offset, dtype=np.uint8)
    dev = torch.from_numpy(frames.copy()).cuda()
    d_imgs = torch.from_numpy(imgs).cuda()
    torch.cuda.synchronize()
    E.encode_2d_image(ctx, d_imgs, (xs, ys), dims, 1.0, dev[offset:], stride)
    ctx.synchronize()
    ref = frames.copy()
    for k in range(n):
        at = offset + k * stride
        one = ref[at:at + dims[0] * dims[1]]
        one[:] = oracle.encode_image(imgs[k], 1.0, *dims, target=one)
    assert np.array_equal(dev.cpu().numpy(), ref)
    ctx.close()
