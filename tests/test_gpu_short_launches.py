"""Staged encodes with and without the block order, on both sides of the number
of blocks where it is left out, and textures whose passes are empty: the blocks
and sums of the single kernel (nebc7_encode_device_noalloc), which the other
tests compare with the oracle."""

import ctypes

import numpy as np
import pytest

from nebc7_gb300 import synth

pytestmark = pytest.mark.gpu

WARPS = 152 * 4 * 4      # resident warps of the staged form on 152 SMs


def texture(kind, blocks_w, blocks_h):
    w, h = 4 * blocks_w, 4 * blocks_h
    if kind == "flat":
        return np.full((h, w, 4), 200, np.uint8)
    img = synth.image_for("photo_like", max(w, 64), max(h, 64), 17)[:h, :w].copy()
    if kind == "half":                        # every other block row of one colour
        img.reshape(blocks_h, 4, w, 4)[::2] = 90
    return np.ascontiguousarray(img)


@pytest.mark.parametrize("kind", ["photo", "flat", "half"])
@pytest.mark.parametrize("blocks", [(1, 1), (1, 5), (64, 37), (64, 38), (61, 40)])
def test_short_launches_equal_the_single_kernel(native, kind, blocks):
    torch = pytest.importorskip("torch")
    from nebc7_gb300._native import Settings
    assert 64 * 38 == WARPS < 61 * 40
    img = texture(kind, *blocks)
    h, w = img.shape[:2]
    d_img = torch.from_numpy(img).cuda()
    stream = torch.cuda.current_stream().cuda_stream
    for st in (Settings(1, 9, 1, 1, 0, 0), Settings(0, 0, 1, 1, 0, 0)):
        assert native.nebc7_init_device(st.denoise) == 0
        a, b = (torch.zeros((w * h // 16, 16), dtype=torch.uint8, device="cuda") for _ in range(2))
        sums = torch.zeros(4, dtype=torch.int64, device="cuda")
        errs, ssim = np.zeros(2, np.int64), np.zeros(2)
        for _ in range(2):      # the second call starts from the first one's blocks
            assert native.nebc7_encode_device(a.data_ptr(), d_img.data_ptr(), None, w * 4, w, h, ctypes.byref(st),
                                              errs.ctypes.data, ssim.ctypes.data, stream) == 0
            assert native.nebc7_encode_device_noalloc(b.data_ptr(), d_img.data_ptr(), None, w * 4, w, h, ctypes.byref(st),
                                                      sums.data_ptr(), stream) == 0
            raw = sums.cpu().numpy()
            assert torch.equal(a, b)
            assert errs.tolist() == raw[:2].tolist() and ssim.tolist() == raw[2:].view(np.float64).tolist()
