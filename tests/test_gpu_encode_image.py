"""encode_image, which pads and masks on the device, against the same steps on
the host (pad_texture, outline_mask, process_texture): ragged sizes down to one
pixel, the outline radii, no mask, starting blocks.  Everything is equal."""

import numpy as np
import pytest

from nebc7_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (3, 5), (4, 4), (37, 2), (65, 130)])
@pytest.mark.parametrize("flags", ["", "/retina", "/nomask", "/draft"])
def test_matches_host_padding(native, w, h, flags):
    from nebc7_gb300 import Bc7Core, Preset, encode_image, outline_mask, pad_texture, parse_flags
    rng = synth.SplitMix64(w * 1000 + h)
    img = rng.below(256, w * h * 4).reshape(h, w, 4).astype(np.uint8)
    img[..., 3][rng.below(3, w * h).reshape(h, w) > 0] = 0
    o = parse_flags(flags)
    padded = pad_texture(img)
    ph, pw = padded.shape[:2]
    core = Bc7Core(Preset(1, 9))
    core.init_tables(o["draft"], o["normal"], o["slow"], o["linear"])
    want = np.zeros((ph * pw // 16, 16), np.uint8)
    stats = core.process_texture(want, padded, outline_mask(padded, o["radius"]) if o["mask"] else None, pw, ph)
    got = encode_image(img[:, ::1], flags, Preset(1, 9))
    assert (got.blocks == want).all() and got.stats == stats
    again = encode_image(img, flags, Preset(1, 9), start=want)
    core.process_texture(want, padded, outline_mask(padded, o["radius"]) if o["mask"] else None, pw, ph)
    assert (again.blocks == want).all()
