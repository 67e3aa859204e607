"""The staged encode when its rooms run out: results that are not kept, blocks
without a place in a later round, estimates that are not handed over, and the
blocks that come back to the one-warp remainder of every split pass (of modes 2
and 0 with the estimates they were handed).  Against the CPU oracle port; blocks
and integer error sums are bit-exact."""

import ctypes

import numpy as np
import pytest

from nebc7_gb300 import synth

pytestmark = pytest.mark.gpu

#          results, later rounds, handed blocks
ROOMS = [(0, -1, -1), (5, -1, -1), (-1, 0, -1), (-1, 3, -1), (-1, -1, 0), (-1, -1, 3), (2, 1, 5), (0, 0, 0)]


def cells(kind, n, seed):
    """Pixels of two or three regions (halves, corners, stripes), each on a line
    of its own, with noise: blocks whose searches improve more than once; or of
    two colours anywhere in the block with little noise (modes 1 and 3), and of a
    few levels (mode 5)."""
    rng = synth.SplitMix64(seed)
    if kind == "two":
        amp = np.array([3, 8, 0])[np.arange(n) % 3][:, None, None]
        part, ends = rng.below(2, n * 16).reshape(n, 16, 1), rng.below(256, n * 8).reshape(n, 2, 4)
        px = np.take_along_axis(ends, part, 1) + rng.below(1 << 16, n * 64).reshape(n, 16, 4) % (2 * amp + 1) - amp
        px[2::3] = 100 + rng.below(12, px[2::3].size).reshape(px[2::3].shape)
        px[:, :, 3] = 255
        return np.clip(px, 0, 255).reshape(n, 64).astype(np.uint8), np.full((n, 64), 255, np.uint8)
    y, x = np.divmod(np.arange(16), 4)
    regions = np.stack([x // 2, y // 2, (x + y) // 3, (x > 1) + (x > 1) * (y > 1), (y > 0) * 1 + (y > 2), (x * y) // 4, x % 2,
                        (x == y) * 1 + (x > y)])[np.arange(n) % 8] % 3
    ends = rng.below(256, n * 24).reshape(n, 3, 2, 4)
    t = rng.below(16, n * 16).reshape(n, 16, 1) / 15.0
    a, b = (np.take_along_axis(ends[:, :, i], regions[:, :, None], 1) for i in (0, 1))
    amp = np.array([2, 6, 12, 40])[np.arange(n) // 8 % 4][:, None, None]
    px = np.clip(np.rint(a + (b - a) * t * 0.4) + rng.below(1 << 16, n * 64).reshape(n, 16, 4) % (2 * amp + 1) - amp, 0, 255)
    if kind == "opaque":
        px[:, :, 3] = 255
    return px.reshape(n, 64).astype(np.uint8), np.full((n, 64), 255, np.uint8)


@pytest.mark.parametrize("kind,n", [("opaque", 32), ("alpha", 32), ("two", 48)])
@pytest.mark.parametrize("denoise,step,slow", [(1, 9, 0), (0, 0, 0), (1, 9, 1), (0, 0, 1)])
def test_blocks_without_room_match_oracle(native, port, kind, n, denoise, step, slow):
    from nebc7_gb300._native import Settings
    c, m = cells(kind, n, 500 + n)
    st = Settings(denoise, step, 1, 1, slow, 0)
    want = np.zeros((n, 16), np.uint8)
    errors, _ = port.compress_blocks(c, m, want, denoise, step, 1, 1, slow, 0, threads=16)
    try:
        for rooms in ROOMS:
            assert native.nebc7_limit_staged_rooms(*rooms) == 0
            got, e = np.zeros((n, 16), np.uint8), np.zeros(2, np.int64)
            assert native.nebc7_encode_blocks_host(c.ctypes.data, m.ctypes.data, got.ctypes.data, n, ctypes.byref(st),
                                                   e.ctypes.data, None) == 0
            bad = np.nonzero((got != want).any(1))[0]
            assert len(bad) == 0, f"rooms {rooms}: {len(bad)} blocks differ, first {bad[:8].tolist()}"
            assert e.tolist() == errors.tolist(), rooms
    finally:
        native.nebc7_limit_staged_rooms(-1, -1, -1)
