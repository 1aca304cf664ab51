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


def test_frames_from_anywhere_are_the_same(of, cuda):
    """Device frames at 16-byte boundaries, at odd pixels, and host frames, of
    more streams than one copy launch takes and of sizes off its 8 pixels."""
    import torch
    base = dataclasses.replace(of.CONFIGS["c1"], resolution=32, max_depth_mm=4000.0)
    cfgs = [dataclasses.replace(base, width=w, height=h, cx=w / 2, cy=h / 2)
            for w, h in ((17, 13), (24, 18), (40, 31))]
    cfgs = [cfgs[i % 3] for i in range(131)]
    rng = np.random.default_rng(0)
    host = [[torch.from_numpy(rng.integers(400, 3000, (c.height, c.width)).astype(np.int16)) for c in cfgs]
            for _ in range(2)]

    def shifted(t):
        buf = torch.zeros(t.numel() + 1, dtype=torch.int16, device=cuda)
        buf[1:] = t.reshape(-1).to(cuda)
        return buf[1:]

    out = []
    for place in (lambda t: t.to(cuda), shifted, lambda t: t):
        b = of.Batch(cfgs, [np.eye(4)] * len(cfgs), use_graph=False)
        frames = []
        for k in range(2):
            depth = [place(t) for t in host[k]]
            b.process(depth)
            torch.cuda.synchronize()
            for i, c in enumerate(cfgs):
                got = torch.as_tensor(_Words(b.buffers(i).depth, c.width * c.height), device=cuda)
                frames.append(got.cpu())
                assert torch.equal(frames[-1], host[k][i].reshape(-1))
        out.append(b.poses())
        b.close()
    assert np.array_equal(out[0], out[1], equal_nan=True) and np.array_equal(out[0], out[2], equal_nan=True)


class _Words:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i2", "data": (int(ptr), False),
                                         "version": 3}
