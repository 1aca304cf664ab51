"""The one-launch filter chain at the edges of its tiles (64 x 17) against the
oracle's filters applied one after another, bit for bit: images smaller than a
tile, one pixel short of, at and past its multiples, odd widths, every mix of
the 16-bit steps, another null value, depths up to 65535, and a frame of nulls
and values that tie."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHAINS = [(("median5",), 1), (("gradient",), 1), (("average",), 4), (("median5", "average"), 1),
          (("median5", "gradient", "average"), 4)]


@pytest.mark.parametrize("w,h", [(8, 8), (63, 16), (64, 17), (65, 18), (131, 35)])
@pytest.mark.parametrize("nullv", [0, 65535, 700])
def test_chains_match_oracle_step_by_step(of, ora, cuda, w, h, nullv):
    import torch
    cfg = dataclasses.replace(of.CONFIGS["c1"], width=w, height=h, cx=w / 2, cy=h / 2)
    rng = np.random.default_rng([w, h, nullv])
    smooth = 700 + 3 * np.arange(w)[None, :] + 2 * np.arange(h)[:, None] + rng.integers(0, 6, (h, w))
    wild = rng.choice([0, 1, 700, 701, 65534, 65535], (h, w))
    for d in (smooth.astype(np.uint16), wild.astype(np.uint16)):
        d[rng.random(d.shape) < 0.3] = nullv
        for steps, passes in CHAINS:
            ref = d
            for step in steps:
                for _ in range(passes if step == "average" else 1):
                    thr = {"average": 15.0, "gradient": 10.0}.get(step, 0.0)
                    ref, _ = ora.depth_filter(step, ref, null_value=nullv, thr=thr)
            t = torch.from_numpy(d.view(np.int16)).to(cuda)
            got = of.depth_filter(cfg, t, steps, null_value=nullv, average_passes=passes)
            assert np.array_equal(got.cpu().numpy().view(np.uint16), ref), (steps, passes)
            of.depth_filter(cfg, t, steps, out=t, null_value=nullv, average_passes=passes)
            assert np.array_equal(t.cpu().numpy().view(np.uint16), ref), (steps, passes, "in place")
