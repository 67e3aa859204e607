"""The combination searches and candidate scans where they can go wrong,
against the CPU oracle port: noise blocks whose lists are full, every count of
visible pixels (rows of a plane come in fours), masks that keep the bounds
lower bounds and masks that do not, flat channels and ranges at the ends of
the value scale.  Blocks and integer error sums are bit-exact."""

import ctypes

import numpy as np
import pytest

from nebc7_gb300 import synth

pytestmark = pytest.mark.gpu


def cells(kind, n, seed):
    rng = synth.SplitMix64(seed)
    px = rng.below(256, n * 64).reshape(n, 16, 4)
    mask = np.full((n, 16, 4), 255, np.int64)
    if kind == "opaque":
        px[:, :, 3] = 255
    elif kind == "visible":            # 0..16 visible pixels, the others alpha-only
        px[:, :, :3] = 96 + px[:, :, :3] % 64
        hidden = np.arange(16)[None, :] >= (np.arange(n) % 17)[:, None]
        mask[:, :, 1:][hidden] = 0
        px[:, :, 3][hidden] = 0
    elif kind == "partial":            # colour channels masked one by one
        px[:, :, :3] = 96 + px[:, :, :3] % 64
        mask[:, :, 2:] = np.where(rng.below(3, n * 32).reshape(n, 16, 2) == 0, 0, 255)
    elif kind == "flat":               # one to four values a channel, at the ends of the scale
        vals = np.array([0, 1, 254, 255])
        px = vals[px % (1 + np.arange(n)[:, None, None] % 4)]
        px[::2, :, 3] = 255
    return (px.reshape(n, 64).astype(np.uint8), mask.reshape(n, 64).astype(np.uint8))


@pytest.mark.parametrize("kind,n", [("opaque", 10), ("visible", 34), ("partial", 32), ("flat", 12)])
@pytest.mark.parametrize("preset,slow,linear", [((1, 9), 0, 0), ((1, 9), 1, 0), ((0, 0), 1, 0), ((1, 9), 0, 1)])
def test_searches_match_oracle(native, port, kind, n, preset, slow, linear):
    from nebc7_gb300._native import Settings
    c, m = cells(kind, n, 77 + n)
    st = Settings(preset[0], preset[1], 1, 1, slow, linear)
    a, b = np.zeros((n, 16), np.uint8), np.zeros((n, 16), np.uint8)
    e1, _ = port.compress_blocks(c, m, a, preset[0], preset[1], 1, 1, slow, linear, threads=16)
    e2 = np.zeros(2, np.int64)
    assert native.nebc7_encode_blocks_host(c.ctypes.data, m.ctypes.data, b.ctypes.data, n, ctypes.byref(st), e2.ctypes.data,
                                           None) == 0
    bad = np.nonzero((a != b).any(1))[0]
    assert len(bad) == 0, f"{len(bad)} blocks differ, first {bad[:8].tolist()}"
    assert e1.tolist() == e2.tolist()
