"""Tone mapping starts beside the end of the work before it on its stream but reads
its input only after it: images written just before on the same stream (by a
kernel, a copy, another tone mapping's bytes), with ragged sizes and several turns
a thread, captured and direct, against the step table."""
import numpy as np
import pytest
import torch

from crisoptix_b200 import _abi, image
import ctypes

pytestmark = pytest.mark.gpu


def table():
    t, c = np.zeros(256, np.float32), ctypes.c_float()
    _abi.check(_abi.load().crisb_srgb8_thresholds(t.ctypes.data_as(ctypes.c_void_p), ctypes.byref(c)))
    return t, c.value


def expected(x):
    t, c_max = table()
    b = np.searchsorted(t[1:], x, side="right").astype(np.uint8)
    return np.where((x >= 0) & (x <= c_max), b, 0).astype(np.uint8)


@pytest.mark.parametrize("pixels", [1, 3, 2048, 2051, 1184 * 512 * 4 + 5, 3 * 592 * 512 * 4 + 1])
@pytest.mark.parametrize("captured", [False, True])
def test_reads_what_the_work_before_wrote(cuda_device, pixels, captured):
    rng = torch.Generator(device="cuda").manual_seed(pixels)
    a = torch.randn(pixels, 3, device="cuda", generator=rng).mul_(0.5)
    x, out = torch.zeros_like(a), torch.zeros(pixels, 3, dtype=torch.uint8, device="cuda")
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    image.tonemap(x, out, st.cuda_stream)  # the table's upload, outside a capture
    torch.cuda.synchronize()
    got = []

    def chain():
        for k in range(4):
            torch.mul(a, 1.0 + k, out=x)
            image.tonemap(x, out, st.cuda_stream)
            got.append(out.clone())

    with torch.cuda.stream(st):
        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st):
                chain()
            g.replay()
        else:
            chain()
    torch.cuda.synchronize()
    h = a.cpu().numpy()
    for k, o in enumerate(got):
        assert np.array_equal(o.cpu().numpy(), expected(h * np.float32(1.0 + k))), k
