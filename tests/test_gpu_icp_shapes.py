"""The single-stream ICP kernel's shapes: frame pyramids on and off a 32-byte
boundary (one load a point, or two), a level whose points fill less than a
chain, and an image whose points exceed a block's shared-memory cache (the
rest is read from memory at every iteration). The pose bar against the FP64
oracle is the other ICP tests' (1e-5 rad, 0.01 mm)."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from conftest import pose_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1280, 960), (203, 157), (24, 18)])
def test_track_matches_oracle_at_any_alignment(of, ora, cuda, w, h):
    import torch
    from openfusion_b200 import _native as N
    base = of.CONFIGS["c2"]
    f = base.fx * w / base.width
    cfg = dataclasses.replace(base, width=w, height=h, fx=f, fy=f, cx=(w - 1) / 2, cy=(h - 1) / 2,
                              resolution=256, trunc_mm=47.0)
    seq = of.make_sequence(cfg, frames=3)
    depth = [torch.from_numpy(d.astype(np.int16)).to(cuda) for d in seq.depth]
    vol, lam = of.new_volume(cfg, cuda), of.lambda_table(cfg, cuda)
    pose = torch.tensor(seq.poses[0].reshape(16), dtype=torch.float64, device=cuda)
    of.integrate(cfg, vol, depth[0], pose, lam)
    model, frame = of.raycast(cfg, vol, pose), of.preprocess(cfg, depth[1])
    ws = of.icp_workspace(cfg, cuda)
    got = pose.clone()
    of.icp_track(cfg, frame, model, got, ws)
    shifted = torch.zeros(frame.numel() + 16, dtype=torch.uint8, device=cuda)
    shifted[16:] = frame
    other = pose.clone()
    cam, icp = cfg.camera(), cfg.icp()
    N.check("of_icp_track", N.lib().of_icp_track(
        C.byref(cam), C.byref(icp), shifted.data_ptr() + 16, model.data_ptr(), other.data_ptr(),
        ws.data_ptr(), None, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(got, other)

    def packed(pyr, with_depth):
        pts, dep = [], []
        for l in range(cfg.levels):
            v, n = of.unpack_points(cfg, pyr, l)
            pts.append(np.concatenate([v.cpu().numpy(), n.cpu().numpy()], -1))
            if with_depth:
                dep.append(of.unpack_depth(cfg, pyr, l).cpu().numpy())
        return ora.pack_pyramid(cfg, pts, dep) if with_depth else ora.pack_pyramid(cfg, pts)

    st, ref, _ = ora.icp_track(cfg, packed(frame, True), packed(model, False), seq.poses[0])
    if st == 0:
        rot, trans = pose_error(got.cpu().numpy().reshape(4, 4), ref)
        assert rot <= 1e-5 and trans <= 1e-2, (rot, trans)
    assert st == 0 or w < 100
