"""Partitions passed over by the principal-axis bound of their subsets, where
it lies closest to the error: the pixels of each half on a line of the four
channels, with noise from none to the rounding slack and past it, and values at
the ends of the scale, whose differences the undenoised error caps.  Against
the CPU oracle port; blocks and integer error sums are bit-exact."""

import ctypes

import numpy as np
import pytest

from nebc7_gb300 import synth

pytestmark = pytest.mark.gpu


def blocks(kind, n, seed):
    rng = synth.SplitMix64(seed)
    if kind == "extremes":
        px = rng.below(2, n * 64).reshape(n, 16, 4) * 255
        px[::3] = np.where(rng.below(8, px[::3].size).reshape(px[::3].shape) == 0, 128, px[::3])
    else:
        ends = rng.below(256, n * 16).reshape(n, 2, 2, 4)
        half = np.arange(16) % 4 // 2                       # left and right columns
        t = (np.arange(16) * 5 % 16)[None, :, None] / 15.0
        a, b = ends[:, 0][:, half], ends[:, 1][:, half]
        amp = np.array([0, 1, 4, 24])[np.arange(n) % 4][:, None, None]
        noise = rng.below(1 << 16, n * 64).reshape(n, 16, 4) % (2 * amp + 1) - amp
        px = np.clip(np.rint(a + (b - a) * t) + noise, 0, 255)
    return px.reshape(n, 64).astype(np.uint8), np.full((n, 64), 255, np.uint8)


@pytest.mark.parametrize("kind,n", [("lines", 32), ("extremes", 9)])
@pytest.mark.parametrize("denoise,step,slow", [(1, 9, 0), (1, 9, 1), (0, 0, 1)])
def test_bounded_partitions_match_oracle(native, port, kind, n, denoise, step, slow):
    from nebc7_gb300._native import Settings
    c, m = blocks(kind, n, 300 + n)
    st = Settings(denoise, step, 1, 1, slow, 0)
    a, b = np.zeros((n, 16), np.uint8), np.zeros((n, 16), np.uint8)
    e1, _ = port.compress_blocks(c, m, a, denoise, step, 1, 1, slow, 0, threads=16)
    e2 = np.zeros(2, np.int64)
    assert native.nebc7_encode_blocks_host(c.ctypes.data, m.ctypes.data, b.ctypes.data, n, ctypes.byref(st), e2.ctypes.data,
                                           None) == 0
    bad = np.nonzero((a != b).any(1))[0]
    assert len(bad) == 0, f"{len(bad)} blocks differ, first {bad[:8].tolist()}"
    assert e1.tolist() == e2.tolist()


@pytest.mark.parametrize("n", [1023, 1024, 1030])
def test_long_lists_equal_short_ones(native, n):
    """A list of 1024 blocks or more takes its mode 7 candidates four at a time,
    a shorter one singly: the blocks of one call equal those of calls of a third."""
    from nebc7_gb300._native import Settings
    rng = synth.SplitMix64(n)
    c = (96 + rng.below(64, n * 64)).reshape(n, 64).astype(np.uint8)
    m = np.full((n, 64), 255, np.uint8)
    st = Settings(1, 9, 1, 1, 0, 0)

    def encode(lo, hi):
        out = np.zeros((hi - lo, 16), np.uint8)
        cc, mm = np.ascontiguousarray(c[lo:hi]), np.ascontiguousarray(m[lo:hi])
        e = np.zeros(2, np.int64)
        assert native.nebc7_encode_blocks_host(cc.ctypes.data, mm.ctypes.data, out.ctypes.data, hi - lo, ctypes.byref(st),
                                               e.ctypes.data, None) == 0
        return out, e

    whole, errors = encode(0, n)
    cuts = [0, n // 3, 2 * n // 3, n]
    parts = [encode(a, b) for a, b in zip(cuts, cuts[1:])]
    assert (whole == np.concatenate([p[0] for p in parts])).all()
    assert (errors == sum(p[1] for p in parts)).all()


@pytest.mark.parametrize("denoise,step", [(1, 9), (0, 0)])
def test_bounds_beside_option_pca(native, port, denoise, step):
    """OPTION_PCA's own bounds may exceed the errors, so a line bound may only
    end a partition by itself, not together with one of them."""
    from nebc7_gb300._native import Settings
    n = 24
    c, m = blocks("lines", n, 911)
    c.reshape(n, 16, 4)[..., 3] = 255
    a, b = np.zeros((n, 16), np.uint8), np.zeros((n, 16), np.uint8)
    assert native.nebc7_set_pca(1) == 0
    port.lib.nebc7_oracle_set_pca(1)
    try:
        e1, _ = port.compress_blocks(c, m, a, denoise, step, 1, 1, 1, 0, threads=16)
        e2 = np.zeros(2, np.int64)
        st = Settings(denoise, step, 1, 1, 1, 0)
        assert native.nebc7_encode_blocks_host(c.ctypes.data, m.ctypes.data, b.ctypes.data, n, ctypes.byref(st), e2.ctypes.data,
                                               None) == 0
    finally:
        native.nebc7_set_pca(0)
        port.lib.nebc7_oracle_set_pca(0)
    assert (a == b).all() and e1.tolist() == e2.tolist()
