"""The light stage without indirect shadow (VPLs staged in shared memory, a
warp per cache and chunk of VPLs) against the FP64 gather with full visibility,
at VPL counts below a round of 32, across light boundaries inside a chunk,
over several chunks, and beyond what shared memory stages. Tolerances: FP32
rounding of a few thousand products (1e-5 relative L2), or BF16 storage (each
coefficient within 2^-9 of itself: 4e-3)."""
import numpy as np
import pytest

from dynamicradiancevolume_gb300 import abi, pipeline
from test_gpu_parity import Run, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("lights,rsm,sh,caches", [(1, 4, 1, 8192), (3, 8, 2, 8192), (2, 32, 2, 8192), (1, 64, 1, 700),
                                                  (3, 64, 2, 8192)])
def test_unshadowed_stage_matches_fp64(lights, rsm, sh, caches, bf16, lib, oracle, cuda):
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=96, height=64, n_lights=lights, rsm_resolution=rsm,
                        indirect_shadow=0, sh_order=sh, max_caches=caches,
                        precision=abi.PRECISION_BF16 if bf16 else abi.PRECISION_FP32)
    r = Run(w, oracle, seed=17)
    n = r.positions.shape[0]
    assert n > 100
    ref = oracle.light_caches_shadowed(r.hf.config, r.positions.copy(), r.hf.lights, r.gpu_vpls_f64(),
                                       np.ones((n, lights * rsm * rsm)))
    assert np.abs(ref).max() > 0
    nk = 27 if sh == 2 else 12
    assert rel_l2(r.gpu_sh()[:, :nk], ref[:, :nk]) < (4e-3 if bf16 else 1e-5)
    # lit again from the same state: the sums are added once more, the same bits each time
    if not bf16:
        r.pipe.light()
        r.pipe.sync()
        assert rel_l2(r.pipe.read_entries_decoded(n)[1], 2 * r.gpu_sh()) < 1e-6
    r.pipe.close()
