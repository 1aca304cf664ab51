"""of_mesh_extract where its work split can go wrong, against the FP64
marching-tetrahedra oracle on random volumes: a single brick, volumes whose
brick count is no power of two, cells next to unobserved voxels and to the
volume's far faces, every sign pattern of a cell, and a volume with more
bricks than the blocks look through at once.

Vertices: FP32 interpolation against FP64, coordinates below 1000 mm (one ulp
6e-5 mm) and an interpolation weight off by a few ulp of 1 over an edge of at
most 126 mm (3e-5 mm): 1e-3 mm, the bar of the other mesh test, is far above.
"""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random_volume(of, n, storage, seed):
    cfg = dataclasses.replace(of.CONFIGS["c1"], resolution=n, size_mm=1000.0, storage=storage)
    rng = np.random.default_rng(seed)
    v = rng.uniform(-1.0, 1.0, (n, n, n))
    q = np.round(v * 32767).astype(np.int16) if storage == "i16" else v.astype(np.float16)
    weight = (rng.random((n, n, n)) < 0.97).astype(np.uint16)
    return cfg, of.linear_to_volume(cfg, q.view(np.uint16), weight)


def _oracle(of, ora, cfg, vol):
    q, w = of.volume_to_linear(cfg, vol)
    return ora.mesh(cfg, (q.astype(np.uint32) | (w.astype(np.uint32) << 16)).reshape(-1))


@pytest.mark.parametrize("n,storage", [(8, "i16"), (16, "f16"), (40, "i16")])
def test_random_volumes_match_oracle(of, ora, cuda, n, storage):
    import torch
    cfg, vol = _random_volume(of, n, storage, n)
    tris, ids = of.extract_mesh(cfg, torch.from_numpy(vol).to(cuda), with_ids=True)
    o, oi = _oracle(of, ora, cfg, vol)
    gi = ids.cpu().numpy().astype(np.uint64)
    order = np.argsort(gi)
    assert np.array_equal(gi[order], oi)
    g = tris.cpu().numpy().astype(np.float64)[order]
    perms = [(0, 1, 2), (1, 2, 0), (2, 0, 1), (0, 2, 1), (2, 1, 0), (1, 0, 2)]
    d = np.min([np.abs(g[:, list(p)] - o).max(axis=(1, 2)) for p in perms], axis=0)
    assert d.max() < 1e-3, d.max()
    # a short buffer holds whole triangles of the mesh, each once
    cap = len(oi) // 3
    part, pid = of.extract_mesh(cfg, torch.from_numpy(vol).to(cuda), max_triangles=cap, with_ids=True)
    pid = pid.cpu().numpy().astype(np.uint64)
    assert len(np.unique(pid)) == cap and np.isin(pid, oi).all()
    at = np.searchsorted(oi, pid)
    assert np.array_equal(part.cpu().numpy().astype(np.float64), g[at])


def test_more_bricks_than_one_look(of, ora, cuda):
    """A 24^3 volume in the far corner of a 1024^3 one: the same cells."""
    import torch
    cfg, vol = _random_volume(of, 24, "i16", 3)
    _, oi = _oracle(of, ora, cfg, vol)
    big = dataclasses.replace(cfg, resolution=1024)
    words = of.new_volume(big, cuda)
    bricks = words[:1024 ** 3].view(128, 128, 128, 512)
    bricks[125:, 125:, 125:] = torch.from_numpy(vol[:24 ** 3].reshape(3, 3, 3, 512)).to(cuda)
    flags = words[1024 ** 3:].view(torch.uint8)[:128 ** 3].view(128, 128, 128)
    flags[124:, 124:, 124:] = 1
    _, ids = of.extract_mesh(big, words, with_ids=True)
    gi = np.sort(ids.cpu().numpy())
    cell, piece = oi.astype(np.int64) // 12, oi.astype(np.int64) % 12
    i, j, k = cell // 576 + 1000, (cell // 24) % 24 + 1000, cell % 24 + 1000
    assert np.array_equal(gi, np.sort(((i * 1024 + j) * 1024 + k) * 12 + piece))
