"""drv_frame against the stages called one by one: the frame clears the pair
counters on a side stream, lets the light stage write the dispatch size and
starts the apply on that stage's tail. Shadowed and unshadowed, one light and
three, one frame after another on one context, and a frame without geometry
(every apply thread discards). The sums are FP32 over the same terms; only their
order may differ (1e-5 relative L2)."""
import numpy as np
import pytest

from dynamicradiancevolume_gb300 import abi, pipeline
from test_gpu_parity import rel_l2

pytestmark = pytest.mark.gpu


def _counter(p):
    return list(p._dev_tensor(p.buffers().counter, 4, p.torch.int32).cpu().numpy())


@pytest.mark.parametrize("lights,shadow,per_light,single", [(1, 1, 0, 0), (3, 1, 0, 0), (3, 1, 1, 0), (3, 0, 0, 0),
                                                            (1, 1, 0, 1)])
def test_frame_matches_its_stages(lights, shadow, per_light, single, lib, cuda):
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=101, height=67, n_lights=lights, rsm_resolution=16,
                        indirect_shadow=shadow)
    p = pipeline.Pipeline(pipeline.host_frame(w, seed=11))
    p.set_tuning(per_light_dispatch=per_light, light_path=abi.LIGHT_PATH_SINGLE if single else abi.LIGHT_PATH_SPLIT)
    p.raycast_inputs()
    p.prepare_and_extract()
    p.voxelize()
    p.allocate()
    p.light()
    p.apply()
    p.sync()
    ref, ref_counter = p.out.cpu().numpy().copy(), _counter(p)
    assert ref_counter[0] > 0 and np.abs(ref).max() > 0
    depth = p.depth.clone()
    for _ in range(2):
        p.out.fill_(7.0)
        p.torch.cuda.synchronize()
        p.frame()
        p.sync()
        assert _counter(p) == ref_counter
        assert rel_l2(p.out.cpu().numpy(), ref) < 1e-5
        # no geometry: no cache, black
        p.depth.zero_()
        p.torch.cuda.synchronize()
        p.frame()
        p.sync()
        assert _counter(p) == [0, 1, 1, 0]
        assert not p.out.any()
        p.depth.copy_(depth)
    p.close()
