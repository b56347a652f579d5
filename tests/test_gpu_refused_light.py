"""A frame with a light that is refused: the lights before it are prepared and
extracted all the same, as by the calls per light, so that an extraction called
afterwards reads a chain of this frame's RSM and not an earlier frame's."""
import ctypes as C

import numpy as np
import pytest

from dynamicradiancevolume_gb300 import abi, pipeline

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("refuse", ["view", "interval"])
def test_lights_before_a_refused_one_are_prepared(refuse, lib, cuda):
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=64, height=64, n_lights=2, rsm_resolution=32,
                        rsm_read_lod=2)
    p = pipeline.Pipeline(pipeline.host_frame(w, 1))
    p.raycast_inputs()
    p.prepare_and_extract()
    p.sync()
    first = p.read_vpls(0).cpu().numpy()
    p.set_frame(pipeline.host_frame(w, 2))
    p.raycast_inputs()
    p.prepare_and_extract()
    p.sync()
    second = p.read_vpls(0).cpu().numpy()
    assert not np.array_equal(first, second)
    p.set_frame(pipeline.host_frame(w, 1))
    p.raycast_inputs()
    p.frame()
    p.sync()
    assert np.array_equal(p.read_vpls(0).cpu().numpy(), first)
    p.set_frame(pipeline.host_frame(w, 2))
    p.raycast_inputs()
    if refuse == "view":
        p.rsm_views[1].resolution = 0
    else:
        p.hf.lights[1].indirect_shadow_sample_interval = 0
    st = lib.drv_frame(p.ctx, C.byref(p.hf.scene), C.byref(p.gview), C.byref(p.hf.frame), C.byref(p.hf.volume),
                       p.hf.lights, p.rsm_views, 2, C.c_void_p(p.out.data_ptr()))
    assert st == abi.ERR_INVALID_ARG
    p.sync()
    assert np.array_equal(p.read_vpls(0).cpu().numpy(), second)  # extracted by the frame
    assert lib.drv_extract_vpls(p.ctx, 0, C.byref(p.hf.lights[0])) == abi.OK
    p.sync()
    assert np.array_equal(p.read_vpls(0).cpu().numpy(), second)
    p.close()
