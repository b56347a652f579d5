"""The list of large triangles at each of its lengths: a mesh of large triangles
once (all listed, a few), repeated to some 20 thousand (all listed still: the pass
over the triangles alone would leave most warps idle) and to some 60 thousand (the
list is full, the rest are walked where they were set up). The surfaces are the
same, so depth, normals, albedo, the RSM's flux, normals and distances, and the
voxels are the same bit for bit. How many triangles are large is counted on the
host, so that each form is known to run."""
import numpy as np
import pytest

from dynamicradiancevolume_gb300 import pipeline
from test_gpu_mesh import Mesh, _raster_inputs, _snapshot
from test_gpu_triangles import _gpu_bits

pytestmark = pytest.mark.gpu

DIRECT = 512       # pixels of a bounding box up to which a triangle is not listed
FULL = 16384       # entries of the list for long meshes
LISTS_ALL = 43776  # triangles up to which every large one is listed (152 SMs x 36 warps x 8)


def _large(m, tris, w, h):
    """Triangles wholly in front of the near plane whose clamped box is certainly above DIRECT pixels."""
    c = np.concatenate([tris.astype(np.float64), np.ones(tris.shape[:2] + (1,))], -1) @ np.array(m[:]).reshape(4, 4).T
    front = ((c[..., 3] > 0) & (c[..., 3] >= c[..., 2])).all(-1)
    with np.errstate(divide="ignore", invalid="ignore"):
        s = (c[..., :2] / c[..., 3:] * 0.5 + 0.5) * [w, h]
    lo = np.clip(np.floor(s.min(1)), 0, [w - 1, h - 1])
    hi = np.clip(np.floor(s.max(1)), 0, [w - 1, h - 1])
    hit = front & (s.max(1) >= 0).all(-1) & (s.min(1) < [w, h]).all(-1)
    return int((hit & ((hi - lo - 1).clip(0).prod(-1) > DIRECT)).sum())


def test_each_form_of_the_list_gives_the_same(lib, cuda):
    torch = pytest.importorskip("torch")
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=301, height=203, rsm_resolution=256, voxel_res=128)
    p = pipeline.Pipeline(pipeline.host_frame(w, 5))
    rng = np.random.default_rng(4)
    centre = rng.uniform(0.2, 0.8, (100, 1, 3))
    tris = (centre + rng.uniform(-0.35, 0.35, (100, 3, 3))).astype(np.float32)
    alb = rng.uniform(0.1, 1.0, (100, 3)).astype(np.float32)
    large = [_large(p.hf.frame.view_projection, tris, w.width, w.height),
             _large(p.hf.lights[0].view_projection, tris, w.rsm_resolution, w.rsm_resolution)]
    refs = None
    for copies in (1, 400, 1200):
        n = 100 * copies
        if copies > 1:
            assert min(large) * copies > FULL and (n <= LISTS_ALL) == (copies == 400), (large, n)
        flat = np.tile(tris, (copies, 1, 1)).reshape(-1, 3)
        _raster_inputs(p, lib, Mesh(torch, p.device, flat, None, np.tile(alb, (copies, 1))))
        g, r = _snapshot(p)
        got = [g["depth"], g["normal16"], g["albedo"], *r[0], _gpu_bits(p, flat)]
        assert (g["depth"] > 0).mean() > 0.5 and r[0][0].any()
        refs = refs or got
        for a, b in zip(refs, got):
            assert np.array_equal(a, b)
    p.close()


@pytest.mark.parametrize("size,copies", [(0.02, (1, 100, 101, 201, 850)), (0.2, (1, 26, 27, 201))])
def test_triangles_per_warp_give_the_same(size, copies, lib, cuda):
    """One triangle per warp, two (from 9729 on, 152 SMs x 64 warps), three and eight,
    and the voxels' walk where it was set up and by tiles (boxes of up to some 50
    x 50 voxels, listed above 512 or, from 2432 triangles on, above 4096): the same
    surfaces, so the same images and voxels."""
    torch = pytest.importorskip("torch")
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=217, height=150, rsm_resolution=64, voxel_res=128)
    p = pipeline.Pipeline(pipeline.host_frame(w, 5))
    rng = np.random.default_rng(9)
    tris = (rng.uniform(0.1, 0.9, (97, 1, 3)) + rng.uniform(-size, size, (97, 3, 3))).astype(np.float32)
    alb = rng.uniform(0.1, 1.0, (97, 3)).astype(np.float32)
    refs = None
    for k in copies:
        flat = np.tile(tris, (k, 1, 1)).reshape(-1, 3)
        _raster_inputs(p, lib, Mesh(torch, p.device, flat, None, np.tile(alb, (k, 1))))
        g, r = _snapshot(p)
        got = [g["depth"], g["normal16"], g["albedo"], *r[0], _gpu_bits(p, flat)]
        assert g["depth"].any() and got[-1].any()
        refs = refs or got
        for a, b in zip(refs, got):
            assert np.array_equal(a, b)
    p.close()
