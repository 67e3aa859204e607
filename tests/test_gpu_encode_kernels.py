"""nebc7_encode_kernels against the kernels that an encode enqueues: the kernel
nodes of a captured nebc7_encode_device call (nothing is launched)."""

import ctypes

import numpy as np
import pytest

from nebc7_gb300 import synth

pytestmark = pytest.mark.gpu

KERNEL_NODE = 0      # cudaGraphNodeTypeKernel
RELAXED = 2          # cudaStreamCaptureModeRelaxed


def runtime(torch):
    major = torch.version.cuda.split(".")[0]
    for name in (f"libcudart.so.{major}", "/usr/local/cuda/lib64/libcudart.so"):
        try:
            return ctypes.CDLL(name)
        except OSError:
            pass
    pytest.skip("no CUDA runtime library to capture with")


@pytest.mark.parametrize("side", [192, 256])      # 2304 blocks, a warp each, and 4096
@pytest.mark.parametrize("settings", [(1, 9, 1, 0, 0, 0), (1, 9, 2, 1, 0, 0), (1, 9, 1, 1, 0, 0), (0, 0, 1, 1, 0, 0),
                                      (1, 9, 1, 1, 1, 0), (1, 9, 1, 1, 0, 1)])
def test_kernels_of_a_captured_encode(native, settings, side):
    torch = pytest.importorskip("torch")
    from nebc7_gb300._native import Settings
    cuda = runtime(torch)
    w = h = side
    img = torch.from_numpy(np.ascontiguousarray(synth.image_for("photo_like", w, h, 5))).cuda()
    dst = torch.zeros((w * h // 16, 16), dtype=torch.uint8, device="cuda")
    st = Settings(*settings)
    stream = torch.cuda.Stream()
    handle = ctypes.c_void_p(stream.cuda_stream)

    def encode():
        return native.nebc7_encode_device(dst.data_ptr(), img.data_ptr(), None, w * 4, w, h, ctypes.byref(st), None, None, handle)

    assert encode() == 0      # builds the tables
    torch.cuda.synchronize()
    graph, n = ctypes.c_void_p(), ctypes.c_size_t()
    assert cuda.cudaStreamBeginCapture(handle, RELAXED) == 0
    rc = encode()
    assert cuda.cudaStreamEndCapture(handle, ctypes.byref(graph)) == 0 and rc == 0
    try:
        assert cuda.cudaGraphGetNodes(graph, None, ctypes.byref(n)) == 0
        nodes = (ctypes.c_void_p * n.value)()
        assert cuda.cudaGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
        kinds = []
        for node in nodes:
            kind = ctypes.c_int()
            assert cuda.cudaGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
            kinds.append(kind.value)
    finally:
        cuda.cudaGraphDestroy(graph)
    kernels = native.nebc7_encode_kernels(ctypes.byref(st))
    ordered = settings[3] and settings[2] != 2       # the refining presets order a long launch's blocks
    assert kinds.count(KERNEL_NODE) == kernels - (2 if ordered and side == 192 else 0)
