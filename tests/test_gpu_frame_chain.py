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


@pytest.mark.parametrize("bf16", [False, True])
def test_lights_of_different_resolutions_share_launches(bf16, lib, cuda):
    """A frame's RSM chains and extractions run all lights per launch, those with
    as many passes left together: the VPLs and shadow cones of lights that read
    different levels of their chains are bit for bit those of the calls per light."""
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=64, height=64, n_lights=4, rsm_resolution=64,
                        rsm_read_lod=0, precision=abi.PRECISION_BF16 if bf16 else abi.PRECISION_FP32)
    p = pipeline.Pipeline(pipeline.host_frame(w, seed=2))
    p.raycast_inputs()
    for l, (read, shadow_lod) in enumerate([(64, 0), (4, 1), (16, 1), (8, 0)]):  # 0, 5, 3 and 3 passes
        p.hf.lights[l].rsm_read_resolution = read
        p.hf.lights[l].indirect_shadow_lod = shadow_lod
        p.hf.lights[l].indirect_shadow_sample_interval = 4 ** shadow_lod
    p.prepare_and_extract()
    p.sync()

    def state():
        b = p.buffers()
        return [(p._dev_tensor(b.vpls[l], b.n_vpls[l] * (8 if bf16 else 12), p.torch.int32).cpu().numpy(),
                 p._dev_tensor(b.cones[l], b.n_vpls[l] // 4 ** shadow * 4, p.torch.int32).cpu().numpy())
                for l, shadow in enumerate((0, 1, 1, 0))]

    ref = state()
    p.frame()
    p.sync()
    got = state()
    for (v0, c0), (v1, c1) in zip(ref, got):
        assert np.any(v0) and np.array_equal(v0, v1) and np.array_equal(c0, c1)
    p.close()
