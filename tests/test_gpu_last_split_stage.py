"""drv_get_light_pairs reports the last split light stage: a frame that takes the
single-launch form (more shadow blocks than the split stage lists) and a frame
that is refused leave it as it was."""
import ctypes as C

import pytest

from dynamicradiancevolume_gb300 import abi, pipeline

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("other", ["single", "refused"])
def test_other_frames_leave_the_pair_count(other, lib, cuda):
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=24, height=16, rsm_resolution=512, rsm_read_lod=4)
    p = pipeline.Pipeline(pipeline.host_frame(w, 8))
    p.raycast_inputs()
    p.frame()
    p.sync()
    pairs = p.light_pairs()
    assert pairs > 0
    L = p.hf.lights[0]
    if other == "single":
        L.rsm_read_resolution = 512  # 262144 blocks
        p.frame()
    else:
        L.indirect_shadow_sample_interval = 0
        assert lib.drv_frame(p.ctx, C.byref(p.hf.scene), C.byref(p.gview), C.byref(p.hf.frame), C.byref(p.hf.volume),
                             p.hf.lights, p.rsm_views, 1, C.c_void_p(p.out.data_ptr())) == abi.ERR_INVALID_ARG
    p.sync()
    assert p.light_pairs() == pairs
    p.close()
