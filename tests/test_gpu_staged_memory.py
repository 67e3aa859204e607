"""Encodes, batches and servers that find no memory for the staged form's
records: every call is still taken, and its blocks and sums are those of the
staged form (which the other tests compare with the oracle)."""

import ctypes

import numpy as np
import pytest

from nebc7_gb300 import synth

pytestmark = pytest.mark.gpu

PRESETS = {"draft": (1, 9, 1, 0, 0, 0), "default": (1, 9, 1, 1, 0, 0), "precise": (0, 0, 1, 1, 0, 0)}


@pytest.fixture
def limit(native):
    yield lambda n: native.nebc7_limit_staged_records(n)
    native.nebc7_limit_staged_records(-1)


def _image(w, h, seed):
    return np.ascontiguousarray(synth.image_for("photo_like", w, h, seed))


def _host(native, img, preset):
    from nebc7_gb300._native import Settings
    h, w = img.shape[:2]
    dst, e, q = np.zeros((w * h // 16, 16), np.uint8), np.zeros(2, np.int64), np.zeros(2)
    st = Settings(*PRESETS[preset])
    assert native.nebc7_encode_host(dst.ctypes.data, img.ctypes.data, None, w * 4, w, h, ctypes.byref(st), e.ctypes.data,
                                    q.ctypes.data) == 0
    return dst, e, q


def _device(native, torch, img, preset):
    from nebc7_gb300._native import Settings
    h, w = img.shape[:2]
    d = torch.from_numpy(img).cuda()
    dst = torch.zeros((w * h // 16, 16), dtype=torch.uint8, device="cuda")
    e, q = np.zeros(2, np.int64), np.zeros(2)
    st = Settings(*PRESETS[preset])
    assert native.nebc7_encode_device(dst.data_ptr(), d.data_ptr(), None, w * 4, w, h, ctypes.byref(st), e.ctypes.data,
                                      q.ctypes.data, torch.cuda.current_stream().cuda_stream) == 0
    return dst.cpu().numpy(), e, q


@pytest.mark.parametrize("preset", ["default", "precise"])
def test_encodes_without_records(native, limit, preset):
    torch = pytest.importorskip("torch")
    img = _image(64, 48, 3)
    want = _host(native, img, preset)
    limit(0)
    for got in (_host(native, img, preset), _device(native, torch, img, preset)):
        assert np.array_equal(got[0], want[0]) and got[1].tolist() == want[1].tolist() and got[2].tolist() == want[2].tolist()


# bytes for: no group; the default group alone (64 blocks; its mixed launch has 192); all
@pytest.mark.parametrize("bytes_,staged", [(0, (False, False)), (400_000, (False, True)), (-1, (True, True))])
def test_batches_without_records(native, limit, bytes_, staged):
    torch = pytest.importorskip("torch")
    from nebc7_gb300 import Batch, BatchTexture
    from nebc7_gb300._native import Settings
    imgs = [(_image(32, 32, 7), "default"), (_image(64, 32, 8), "draft")]
    want = [_host(native, *i) for i in imgs]
    dev = [(torch.from_numpy(i).cuda(), torch.zeros((i.shape[0] * i.shape[1] // 16, 16), dtype=torch.uint8, device="cuda"))
           for i, _ in imgs]
    limit(bytes_)
    b = Batch([BatchTexture(d.data_ptr(), s.data_ptr(), None, s.shape[1] * 4, s.shape[1], s.shape[0], Settings(*PRESETS[p]))
               for (s, d), (_, p) in zip(dev, imgs)], from_scratch=True)
    for schedule in (0, 1):
        b.set_schedule(schedule)
        b.launch()
        errs, ssim = b.sums()
        # a group without records: two order kernels, the encode, the sums
        assert (b.info()["launches"] > 4 * (schedule + 1)) == staged[schedule]
        for i, (_, d) in enumerate(dev):
            assert np.array_equal(d.cpu().numpy(), want[i][0])
            assert errs[i].tolist() == want[i][1].tolist() and ssim[i].tolist() == want[i][2].tolist()
    b.close()


@pytest.mark.parametrize("bytes_", [0, 200_000, 700_000])
def test_servers_without_records(native, limit, bytes_):
    """No records, those of fewer blocks than some requests have, and of most."""
    from nebc7_gb300 import Server
    from nebc7_gb300._native import Settings
    reqs = [(_image(16 * (1 + i % 4), 16 * (1 + i % 3), 30 + i), list(PRESETS)[i % 3]) for i in range(12)]
    want = [_host(native, *r) for r in reqs]
    limit(bytes_)
    srv = Server(hbm_budget=1 << 20, max_batch=4, streams=2)
    outs = [np.zeros_like(w[0]) for w in want]
    tickets = [srv.submit(img, None, o, Settings(*PRESETS[p])) for (img, p), o in zip(reqs, outs)]
    infos = [srv.wait(t) for t in tickets]
    srv.close()
    for o, i, w in zip(outs, infos, want):
        assert np.array_equal(o, w[0]) and i["errs"] == w[1].tolist() and i["ssim"] == w[2].tolist()
