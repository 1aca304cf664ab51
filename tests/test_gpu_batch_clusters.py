"""The batched ICP's two cluster sizes: 16 CTAs a stream for a few streams, 8
for many. Both deal a level's pixels to the same 4096 chains and add them in
the same order, so a stream tracked in a small batch and in a large one has
the same pose, bit for bit, at image sizes below, at and off the multiples of
the chains (a 3x2 coarse level leaves most chains empty)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(24, 18), (160, 120), (203, 157)])
def test_both_cluster_sizes_give_the_same_poses(of, cuda, w, h):
    import torch
    base = of.CONFIGS["c1"]
    f = base.fx * w / base.width
    cfg = dataclasses.replace(base, width=w, height=h, fx=f, fy=f, cx=(w - 1) / 2, cy=(h - 1) / 2,
                              resolution=64, max_depth_mm=4000.0)
    seqs = [of.make_sequence(dataclasses.replace(cfg, seed=70 + i), frames=4) for i in range(2)]
    depth = [[torch.from_numpy(q.depth[k].astype(np.int16)).to(cuda) for q in seqs] for k in range(4)]
    few = of.Batch([cfg] * 2, [q.poses[0] for q in seqs])          # 16 CTAs a stream
    many = of.Batch([cfg] * 24, [seqs[i % 2].poses[0] for i in range(24)])  # 8 CTAs
    for k in range(4):
        few.process(depth[k])
        many.process([depth[k][i % 2] for i in range(24)])
        (P, sp), (Q, sq) = few.poses(with_stats=True), many.poses(with_stats=True)
        for i in range(24):
            assert np.array_equal(P[i % 2], Q[i]), (k, i)
            assert (sp[i % 2].iterations, sp[i % 2].inliers, sp[i % 2].residual_sq) == \
                (sq[i].iterations, sq[i].inliers, sq[i].residual_sq)
        if w > 100:
            assert all(s.status == 0 for s in sp) and (k == 0 or all(s.inliers > 100 for s in sp))
    few.close()
    many.close()
