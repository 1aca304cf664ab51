"""The raycast's march and its order of tiles: every block shape writes every
pixel of an image that no tile divides, of one tile and of a single tile row
with the same bits; a small camera's rays are the same bits as the same rays of
a larger one (which leaves them to other blocks); rays in an axis plane (a zero
direction component) and rays that miss the volume are covered."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["i16", "f16"])
@pytest.mark.parametrize("w,h", [(203, 157), (37, 8), (8, 8)])
def test_tiles_and_windows_give_the_same_rays(of, cuda, w, h, storage):
    import torch
    base = of.CONFIGS["c2"]
    cfg = dataclasses.replace(base, width=321, height=241, fx=262.5, fy=262.5, cx=160.0, cy=120.0,
                              resolution=256, trunc_mm=47.0, storage=storage, levels=1)
    seq = of.make_sequence(cfg, frames=3)
    vol, lam = of.new_volume(cfg, cuda), of.lambda_table(cfg, cuda)
    for k in range(3):
        of.integrate(cfg, vol, torch.from_numpy(seq.depth[k].astype(np.int16)).to(cuda),
                     torch.tensor(seq.poses[k].reshape(16), dtype=torch.float64, device=cuda), lam)
    straight = np.eye(4)
    straight[:3, 3] = seq.poses[1][:3, 3]
    away = np.eye(4)
    away[2, 3] = -4.0 * cfg.size_mm  # beyond the far side, looking on
    x0, y0 = (321 - w) // 2, (241 - h) // 2
    cfg_w = dataclasses.replace(cfg, width=w, height=h, cx=cfg.cx - x0, cy=cfg.cy - y0)
    for pose, some in ((seq.poses[2], True), (straight, True), (away, False)):
        p = torch.tensor(pose.reshape(16), dtype=torch.float64, device=cuda)
        full = of.raycast(cfg, vol, p)
        vf, nf = of.unpack_points(cfg, full, 0)
        assert bool((vf[..., 3] > 0).any()) == some
        for tile in range(7):
            c = dataclasses.replace(cfg_w, ray_tile=tile)
            out = of.new_pyramid(c, cuda)
            out.fill_(255)
            of.raycast(c, vol, p, out)
            v, n = of.unpack_points(c, out, 0)
            assert torch.equal(v.view(torch.int32), vf[y0:y0 + h, x0:x0 + w].contiguous().view(torch.int32))
            assert torch.equal(n.view(torch.int32), nf[y0:y0 + h, x0:x0 + w].contiguous().view(torch.int32))
