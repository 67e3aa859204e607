"""CPU tests of encode_image's host side, over a stand-in for the library that
records what it is given."""

import ctypes

import numpy as np
import pytest

import nebc7_gb300 as nb
from nebc7_gb300 import _native
from nebc7_gb300.api import outline_mask, pad_texture, padded_size


class Library:
    """Answers every entry with `codes` (0 where there is none); keeps the texture
    and the mask that nebc7_encode_host is given."""

    def __init__(self, **codes):
        self.codes, self.calls, self.texture, self.mask = codes, [], None, None

    def __getattr__(self, name):
        def entry(*args):
            self.calls.append(name)
            if name == "nebc7_encode_host":
                dst, src, mask, stride, w, h = args[:6]
                self.texture = np.frombuffer(ctypes.string_at(src, stride * h), np.uint8).reshape(h, w, 4)
                self.mask = np.frombuffer(ctypes.string_at(mask, stride * h), np.uint8).reshape(h, w, 4) if mask else None
                ctypes.memset(dst, 7, w * h)
            return self.codes.get(name, 0)
        return entry


@pytest.fixture
def library(monkeypatch):
    def use(**codes):
        lib = Library(**codes)
        monkeypatch.setattr(_native, "load", lambda path=None: lib)
        return lib
    return use


@pytest.mark.parametrize("flags,radius", [("", 1), ("/nomask", -1), ("/retina", 2)])
def test_without_device_memory_for_the_raw_image_the_host_pads(library, flags, radius):
    lib = library(nebc7_encode_image_host=_native.ENOMEM)
    img = np.random.default_rng(1).integers(0, 2, (13, 7, 4), dtype=np.uint8) * 200
    enc = nb.encode_image(img, flags)
    assert lib.calls == ["nebc7_init_device", "nebc7_encode_image_host", "nebc7_encode_host"]
    padded = pad_texture(img)
    assert np.array_equal(lib.texture, padded)
    assert (lib.mask is None) if radius < 0 else np.array_equal(lib.mask, outline_mask(padded, radius))
    assert (enc.width, enc.height) == padded_size(7, 13) and (enc.blocks == 7).all()


def test_other_errors_are_raised(library):
    lib = library(nebc7_encode_image_host=2)
    with pytest.raises(nb.NativeError) as e:
        nb.encode_image(np.zeros((4, 4, 4), np.uint8))
    assert e.value.code == 2 and "nebc7_encode_host" not in lib.calls


IMAGE = np.zeros((13, 8, 4), np.uint8)
BLOCKS = np.zeros((8, 16), np.uint8)     # of the 8x16 padded texture


def read_only(a):
    a = a.copy()
    a.flags.writeable = False
    return a


@pytest.mark.parametrize("dst,img", [
    (BLOCKS, IMAGE[:, ::2]), (BLOCKS, IMAGE.astype(np.int32)), (BLOCKS, np.zeros((13, 8, 3), np.uint8)),
    (BLOCKS, np.zeros((13, 8), np.uint8)), (BLOCKS, np.asfortranarray(IMAGE)), (BLOCKS[:7], IMAGE), (BLOCKS[::2], IMAGE),
    (BLOCKS.astype(np.uint16), IMAGE), (read_only(BLOCKS), IMAGE)])
def test_process_image_refuses_what_it_cannot_pass_on(library, dst, img):
    """The library reads and writes through bare pointers."""
    lib = library()
    with pytest.raises(ValueError):
        nb.Bc7Core().process_image(dst, img, 1)
    assert lib.calls == []


def test_process_image_takes_whole_images(library):
    lib = library()
    for dst in (BLOCKS.copy(), np.zeros(200, np.uint8)):
        nb.Bc7Core().process_image(dst, IMAGE, -1)
    assert lib.calls == ["nebc7_encode_image_host"] * 2


def test_starting_blocks_short_of_the_texture_are_refused(library):
    lib = library()
    with pytest.raises(ValueError):
        nb.encode_image(IMAGE, start=BLOCKS[:5])
    nb.encode_image(IMAGE, start=np.asfortranarray(BLOCKS))
    assert lib.calls[-1] == "nebc7_encode_image_host"
