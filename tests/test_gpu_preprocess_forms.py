"""The bilateral filter's two forms (two pixels a thread for images that fill
the GPU, one below) and the pyramid kernel's two stores, against each other
bit for bit."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frame(of, cuda):
    import torch
    d = of.make_sequence(of.CONFIGS["c2"], frames=1).depth[0].astype(np.int16)
    d[np.random.default_rng(1).random(d.shape) < 0.05] = 0
    return torch.from_numpy(d).to(cuda)


@pytest.mark.parametrize("radius", [1, 2, 3, 9, 11, 16])
def test_both_filter_forms_give_the_same_bits(of, cuda, radius):
    """A 640x480 image and its top left corner, an odd 161 x 123: equal where
    a pixel's window lies in both."""
    import torch
    cfg = dataclasses.replace(of.CONFIGS["c2"], radius_px=radius, levels=1)
    d = _frame(of, cuda)
    whole = of.unpack_depth(cfg, of.preprocess(cfg, d))
    part = dataclasses.replace(cfg, width=161, height=123)
    corner = of.unpack_depth(part, of.preprocess(part, d[:123, :161].contiguous()))
    w, h = 161 - radius, 123 - radius
    assert torch.equal(whole[:h, :w], corner[:h, :w])
    assert float((corner > 0).float().mean()) > 0.8


@pytest.mark.parametrize("w,h,levels", [(640, 480, 3), (97, 67, 4), (33, 32, 2), (8, 8, 1)])
def test_pyramid_stores_do_not_depend_on_the_alignment(of, cuda, w, h, levels):
    import torch
    from openfusion_b200 import _native as N
    import ctypes as C
    cfg = dataclasses.replace(of.CONFIGS["c2"], width=w, height=h, levels=levels)
    d = _frame(of, cuda)[:h, :w].contiguous()
    aligned = of.preprocess(cfg, d)
    n = aligned.numel()
    buf = torch.zeros(n + 16, dtype=torch.uint8, device=cuda)
    cam, fp = cfg.camera(), cfg.filter()
    N.check("of_preprocess", N.lib().of_preprocess(
        C.byref(cam), C.byref(fp), d.data_ptr(), w, buf.data_ptr() + 16,
        torch.cuda.current_stream().cuda_stream))
    assert buf.data_ptr() % 32 == 0 and torch.equal(buf[16:], aligned)
