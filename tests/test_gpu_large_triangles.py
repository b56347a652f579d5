"""Large triangles of the mesh passes: listed and walked tile by tile by the
whole GPU, or walked where they were set up when the list is full. A mesh
repeated until the list overflows has the same surfaces as the mesh itself,
so its depth, normals, albedo and voxels are the same bit for bit (a pixel or
voxel that one of the two walks gained or lost would show); the sizes are
odd, so tiles are cut at every border."""
import ctypes as C

import numpy as np
import pytest

from dynamicradiancevolume_gb300 import abi, pipeline
from test_gpu_mesh import Mesh, _box_mesh, _raster_inputs, _snapshot
from test_gpu_triangles import _gpu_bits, _soup

pytestmark = pytest.mark.gpu

LIST = 16384  # entries of the list


@pytest.mark.parametrize("width,height,rsm", [(97, 61, 64), (257, 130, 128)])
def test_full_list_rasters_the_same(width, height, rsm, lib, cuda):
    torch = pytest.importorskip("torch")
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=width, height=height, rsm_resolution=rsm)
    p = pipeline.Pipeline(pipeline.host_frame(w, 5))
    tris, alb = _box_mesh(p.hf)
    rng = np.random.default_rng(3)
    extra = rng.uniform(-0.2, 1.2, (80, 3, 3)).astype(np.float32).reshape(-1, 3)  # across the near plane too
    tris = np.concatenate([tris, extra])
    alb = np.concatenate([alb, np.full((80, 3), 0.5, np.float32)])
    _raster_inputs(p, lib, Mesh(torch, p.device, tris, None, alb))
    g0, r0 = _snapshot(p)
    n = 2 * LIST // (len(tris) // 3) * 4
    _raster_inputs(p, lib, Mesh(torch, p.device, np.tile(tris, (n, 1)), None, np.tile(alb, (n, 1))))
    g1, r1 = _snapshot(p)
    assert (g0["depth"] != 0).all()
    for k in ("depth", "normal16"):
        assert np.array_equal(g0[k], g1[k]), k
    assert np.array_equal(r0[0][1], r1[0][1]) and np.array_equal(r0[0][2], r1[0][2])
    p.close()


@pytest.mark.parametrize("voxels", [32, 64, 256])
def test_full_list_voxelizes_the_same(voxels, lib, cuda, oracle):
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], voxel_res=voxels)
    p = pipeline.Pipeline(pipeline.host_frame(w, 2))
    soup = _soup(np.random.default_rng(7), p.hf.volume, voxels, 200)
    once = _gpu_bits(p, soup)
    assert np.array_equal(once, oracle.voxelize_triangles(soup, None, p.hf.volume, voxels))
    assert np.array_equal(once, _gpu_bits(p, np.tile(soup, (2 * LIST // 40, 1))))
    p.close()
