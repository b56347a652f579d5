"""Indirect specular without indirect shadow: the shadow sample interval of the
lights plays no part. Lights of a deeper shadow lod (intervals of 4 and 16 VPLs)
give the envmaps and the radiance of interval 1, bit for bit: the VPLs are the
same, in the same order, and so is every sum."""
import numpy as np
import pytest

from dynamicradiancevolume_gb300 import abi, pipeline

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("rsm,lights,single", [(16, 3, 0), (128, 1, 0), (16, 2, 1)])
def test_interval_is_ignored_without_shadow(rsm, lights, single, bf16, lib, cuda):
    def frame(shadow_lod):
        w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=72, height=50, n_lights=lights, rsm_resolution=rsm,
                            indirect_shadow=0, shadow_lod=shadow_lod, specular_envmap_size=8,
                            precision=abi.PRECISION_BF16 if bf16 else abi.PRECISION_FP32)
        p = pipeline.Pipeline(pipeline.host_frame(w, 6))
        p.set_tuning(light_path=abi.LIGHT_PATH_SINGLE if single else abi.LIGHT_PATH_AUTO)
        assert p.hf.lights[0].indirect_shadow_sample_interval == 4 ** shadow_lod
        for l in range(lights):
            for c in range(3):  # VPLs with a flux sum below 0.001 are skipped: bright enough for 128^2 of them
                p.hf.lights[l].intensity[c] *= 1000.0
        p.raycast_inputs()
        p.frame()
        p.sync()
        n = p.cache_count()
        order = np.lexsort(p.read_entries_decoded(n)[0].T[::-1])
        got = p.read_specular(n)[order], p.out.cpu().numpy().copy()
        p.close()
        return got

    env, out = frame(0)
    assert env.any() and out.any()
    for lod in (1, 2):
        e, o = frame(lod)
        assert np.array_equal(e, env) and np.array_equal(o, out)
