"""More contributing pairs than 32 bits count: the claims of the caches beyond a
full list must not come round to the list's start, where they would take the
slots of the caches it holds. Both forms of the stage add the same products in
another order: a lane sums about 2000 of them one after the other, sqrt(2000)
roundings of 2^-24 each (2.7e-6), and a few times that is allowed (2e-5)."""
import numpy as np
import pytest

from dynamicradiancevolume_gb300 import abi, pipeline
from test_gpu_parity import rel_l2

pytestmark = pytest.mark.gpu


def test_more_pairs_than_32_bits(lib, cuda):
    # 65536 VPLs in an empty room and some 10^5 caches all over it: nearly every
    # VPL with flux faces nearly every cache. One cone step: the cones cost little.
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], n_boxes=0, width=144, height=128, n_lights=1,
                        rsm_resolution=256, rsm_read_lod=0, cav_res=256, max_cone_steps=1, max_caches=1 << 18)
    p = pipeline.Pipeline(pipeline.host_frame(w, 3))
    p.raycast_inputs()
    p.sync()
    torch = p.torch
    share = np.random.default_rng(1).uniform(0.05, 1.0, (w.height, w.width)).astype(np.float32)
    p.depth.div_(torch.from_numpy(share).to(p.device)).clamp_(max=0.9)  # reversed-Z: that share of the way to the wall
    torch.cuda.synchronize()
    p.prepare_and_extract()
    p.voxelize()

    def lit(**knobs):
        p.set_tuning(**knobs)
        p.allocate()
        p.light()
        p.sync()
        pos, sh = p.read_entries_decoded(p.cache_count())
        order = np.lexsort(pos.T[::-1])
        return pos[order], sh[order]

    pos1, sh1 = lit(light_path=abi.LIGHT_PATH_SPLIT, pair_capacity=1 << 22)
    assert p.light_pairs() == 0xFFFFFFFF, p.light_pairs()
    pos2, sh2 = lit(light_path=abi.LIGHT_PATH_SINGLE)
    assert np.array_equal(pos1, pos2)
    assert rel_l2(sh1, sh2) < 2e-5
    p.close()
