"""Tone mappings right behind the work that writes what they read and the work that
reads what they write, on images and bytes of any alignment: a kernel, a copy, and
another tone mapping, whose bytes the next launch overwrites or whose image is made
of its bytes."""
import ctypes

import numpy as np
import pytest
import torch

from crisoptix_b200 import _abi
from test_tonemap_stream_gpu import expected

pytestmark = pytest.mark.gpu


def tone(x, out, pixels, st):
    _abi.check(_abi.load().crisb_tonemap_srgb8(x.data_ptr(), out.data_ptr(), pixels, ctypes.c_void_p(st.cuda_stream)))


# whole and broken vectors, more than one turn a thread, every kind of alignment
@pytest.mark.parametrize("pixels", [1, 5, 2049, 1184 * 512 + 3, 4 * 1184 * 512 + 7])
@pytest.mark.parametrize("in_off,out_off", [(0, 0), (1, 0), (0, 1), (3, 3)])
def test_chain(cuda_device, pixels, in_off, out_off):
    n = 3 * pixels
    gen = torch.Generator(device="cuda").manual_seed(pixels)
    src = [torch.randn(n, device="cuda", generator=gen).mul_(0.7) for _ in range(3)]
    x = torch.zeros(n + in_off, device="cuda")[in_off:]
    y = torch.zeros(n + in_off, device="cuda")[in_off:]
    a = torch.full((n + out_off + 5,), 77, dtype=torch.uint8, device="cuda")
    b, c = torch.zeros_like(a), torch.zeros_like(a)
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        for s in src:
            torch.mul(s, 0.5, out=x)                          # a kernel writes the image
            tone(x, a[out_off:], pixels, st)
            tone(x, b[out_off:], pixels, st)                  # two tone mappings back to back
            torch.div(a[out_off:out_off + n], 255.0, out=y)   # an image made of a tone mapping's bytes
            tone(y, c[out_off:], pixels, st)
            x.copy_(s)                                        # a copy writes the image a launch before reads
            tone(x, b[out_off:], pixels, st)                  # and the bytes are written again
    torch.cuda.synchronize()
    s = src[-1].cpu().numpy()
    want = expected(s * np.float32(0.5))
    assert np.array_equal(a[out_off:out_off + n].cpu().numpy(), want)
    assert np.array_equal(b[out_off:out_off + n].cpu().numpy(), expected(s))
    y_want = torch.div(torch.from_numpy(want).cuda(), 255.0).cpu().numpy()
    assert np.array_equal(c[out_off:out_off + n].cpu().numpy(), expected(y_want))
    assert (a[:out_off] == 77).all() and (a[out_off + n:] == 77).all()
