"""The allocation against the CPU oracle, bit for bit: ragged and large images
(one pixel per thread and two), depths so noisy that a tile keeps many cells,
cell sizes that are no power of two, transition zones of zero, negative and
overflowing size, one cascade, and more cells than entries."""
import numpy as np
import pytest

from dynamicradiancevolume_gb300 import DrvError, abi, pipeline

pytestmark = pytest.mark.gpu


def _positions(p):
    return sorted(map(tuple, p.tolist()))


@pytest.mark.parametrize("width,height,res,cascades,cell,zone,noise,caches,bf16", [
    (1, 1, 2, 1, 1.0, 1.0, 0.0, 512, False),
    (17, 33, 16, 4, 1.0, 1.0, 0.3, 65536, False),
    (250, 131, 32, 4, 0.9, 1.0, 0.3, 65536, True),
    (250, 131, 32, 3, 1.0, 0.0, 0.05, 65536, False),
    (250, 131, 32, 3, 1.0, -2.0, 0.05, 65536, False),
    (250, 131, 32, 3, 1.0, 1e38, 0.05, 65536, False),
    (250, 131, 128, 2, 1.0, 1.0, 0.3, 500, False),
    (1030, 1009, 64, 4, 1.1, 1.0, 0.1, 131072, False),
    (1030, 1009, 32, 2, 1.0, 1.0, 0.0, 131072, True),
])
def test_allocation_matches_oracle(width, height, res, cascades, cell, zone, noise, caches, bf16, lib, oracle, cuda):
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=width, height=height, cav_res=res, n_cascades=cascades,
                        cascade_transition=2.0, rsm_resolution=8, max_caches=caches,
                        precision=abi.PRECISION_BF16 if bf16 else abi.PRECISION_FP32)
    p = pipeline.Pipeline(pipeline.host_frame(w, seed=3))
    vol = p.hf.volume
    vol.cav_transition_zone_size *= zone
    for c in range(cascades):
        vol.cascades[c].world_voxel_size *= cell
    p.raycast_inputs()
    p.sync()
    rng = np.random.default_rng(5)
    depth = p.depth.cpu().numpy()
    depth = (depth * (1.0 + noise * (rng.random(depth.shape) - 0.5))).astype(np.float32)
    depth[rng.random(depth.shape) < 0.02] = 0.0
    depth[0, 0] = 0.97
    p.depth.copy_(p.torch.from_numpy(depth))
    p.torch.cuda.synchronize()
    for _ in range(2):
        p.allocate()
        p.torch.cuda.synchronize()
        st, atlas, pos, count = oracle.allocate_caches(p.hf.config, vol, p.hf.frame, depth)
        if count > caches:
            with pytest.raises(DrvError, match="more light caches"):
                p.sync()
        else:
            p.sync()
        got = p.read_atlas().cpu().numpy()
        total = int(p._dev_tensor(p.buffers().counter, 4, p.torch.int32)[3])
        assert total == count and count > 0
        assert np.array_equal(got != 0, atlas != 0)
        if count <= caches:
            gpos = p.read_entries_decoded(count)[0]
            assert _positions(gpos) == _positions(pos)
            assert np.array_equal(gpos[got[got != 0] - 1], pos[atlas[atlas != 0].astype(np.int64) - 1])
    p.close()
