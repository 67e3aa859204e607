"""The driver-step kernels at the edges of their tiles, against the oracle
and numpy: decode of blocks of every mode, wide and 4-byte aligned rows;
padding and outline masks around 32- and 256-pixel words and 16-row tiles for
small, word-wide and larger radii; the glitch map on unaligned buffers."""

import numpy as np
import pytest

from nebc7_gb300 import outline_mask, pad_texture, synth

pytestmark = pytest.mark.gpu


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("w,h", [(4, 4), (132, 20), (516, 12)])
@pytest.mark.parametrize("shift", [0, 4])
def test_decode_rows(native, port, w, h, shift):
    import torch
    n = (w // 4) * (h // 4)
    blocks = synth.random_start_blocks(n, 9 + n)
    blocks[:, 0] = np.where(np.arange(n) % 9 < 8, 1 << (np.arange(n) % 9 % 8), 0)   # every mode in turn, and none
    stride = w * 4 + shift
    out = torch.zeros(h * stride + 16 + shift, dtype=torch.uint8, device="cuda")
    d = dev(blocks)
    assert native.nebc7_decode_device(d.data_ptr(), out.data_ptr() + shift, stride, w, h, None) == 0
    got = out.cpu().numpy()[shift:shift + h * stride].reshape(h, stride)[:, :w * 4].reshape(h // 4, 4, w // 4, 16)
    want = port.decompress_blocks(blocks).reshape(h // 4, w // 4, 4, 16).transpose(0, 2, 1, 3)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("w,h", [(1, 1), (31, 15), (33, 17), (255, 33), (257, 16), (290, 50)])
@pytest.mark.parametrize("radius", [-1, 0, 1, 2, 16, 31, 32])
def test_padding_and_outline(native, w, h, radius):
    import torch
    rng = synth.SplitMix64(w * 1000 + h)
    img = rng.below(256, w * h * 4).reshape(h, w, 4).astype(np.uint8)
    img[:, :, 3] = np.where(rng.below(400, w * h).reshape(h, w) < 2, img[:, :, 3] | 1, 0)
    padded = pad_texture(img)
    ph, pw = padded.shape[:2]
    d = dev(img)
    p, m = (torch.full((ph, pw, 4), 7, dtype=torch.uint8, device="cuda") for _ in range(2))
    assert native.nebc7_prepare_device(d.data_ptr(), w * 4, w, h, p.data_ptr(), m.data_ptr(), radius, None) == 0
    assert np.array_equal(p.cpu().numpy(), padded)
    want = outline_mask(padded, radius) if radius >= 0 else np.full_like(padded, 255)
    assert np.array_equal(m.cpu().numpy(), want)


@pytest.mark.parametrize("w,h", [(4, 4), (260, 8), (252, 12)])
@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("linear", [0, 1])
def test_glitch_map(native, w, h, shift, linear):
    import torch
    rng = synth.SplitMix64(w + h)
    src = rng.below(256, w * h * 4).reshape(h, w, 4)
    dec = np.clip(src + rng.between(-22, 22, w * h * 4).reshape(h, w, 4) * (rng.below(12, w * h).reshape(h, w, 1) == 0), 0, 255)
    mask = np.where(rng.below(3, w * h * 4).reshape(h, w, 4) == 0, rng.below(256, w * h * 4).reshape(h, w, 4), 255)
    thr = np.array([16, 16, 16, 16] if linear else [20, 12, 16, 16])   # B, G, R, A
    diff = np.abs(src - dec) & mask[:, :, [3, 1, 2, 0]]
    bad = (diff >= thr).any(2).reshape(h // 4, 4, w // 4, 4).any((1, 3))
    want = np.where(np.repeat(np.repeat(bad, 4, 0), 4, 1)[:, :, None], src, 0).astype(np.uint8)
    bufs = []
    for a in (src, dec, mask, np.zeros_like(src)):
        t = torch.zeros(w * h * 4 + 16, dtype=torch.uint8, device="cuda")
        t[shift:shift + w * h * 4] = dev(a.astype(np.uint8)).flatten()
        bufs.append(t)
    s, d, m, o = (t.data_ptr() + shift for t in bufs)
    assert native.nebc7_bad_blocks_device(s, d, m, w * 4, w, h, linear, o, None) == 0
    assert np.array_equal(bufs[3].cpu().numpy()[shift:shift + w * h * 4].reshape(h, w, 4), want)
