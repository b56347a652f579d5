"""The brute-force gather at the edges of its pixel tiles and VPL batches,
against the FP64 oracle on the GPU's own VPLs: images smaller and one larger
than a tile, VPL counts below and beyond a batch, several lights, both
storage precisions, with and without the reference BRDF. Tolerances as the
full-size tests' (FP32 rounding of a sum of thousands of positive terms); the
oracle reads the stored VPL values, so BF16 storage changes nothing."""
import numpy as np
import pytest

from dynamicradiancevolume_gb300 import abi, pipeline
from test_gpu_parity import Run, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("width,height,lights,rsm", [(1, 1, 1, 8), (31, 17, 2, 16), (33, 16, 1, 32), (65, 39, 3, 32)])
def test_bruteforce_tiles_match_fp64(width, height, lights, rsm, bf16, lib, oracle, cuda):
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=width, height=height, n_lights=lights,
                        rsm_resolution=rsm, indirect_shadow=0, sh_order=2, max_caches=8192,
                        precision=abi.PRECISION_BF16 if bf16 else abi.PRECISION_FP32)
    r = Run(w, oracle, seed=17)
    out = r.pipe.bruteforce().cpu().numpy()
    ref = oracle.bruteforce_rsm(r.hf.frame, r.depth, r.n16, r.albedo, r.gpu_vpls_f64())
    assert np.count_nonzero(ref) > 0
    assert np.all((out == 0) | (ref != 0))  # nothing where no VPL reaches
    assert rel_l2(out, ref) < 1e-5
    rm = np.stack(np.meshgrid(np.linspace(0.2, 1.0, width), np.linspace(0.0, 1.0, height)), -1).astype(np.float32)
    out = r.pipe.bruteforce(rough_metal=r.torch.from_numpy(rm).cuda()).cpu().numpy()
    ref = oracle.bruteforce_rsm(r.hf.frame, r.depth, r.n16, r.albedo, r.gpu_vpls_f64(), rough_metal=rm)
    assert rel_l2(out, ref) < 1e-4
    r.pipe.close()
