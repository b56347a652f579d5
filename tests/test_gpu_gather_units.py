"""The gather's units: runs of one unit and of many, few caches with long runs
and blocks of several VPLs, lit twice (the sums are added once more), and a pair
list that holds part of the caches — against the single-launch form. Tolerances:
FP32 sums of a few thousand products in another order (1e-5 relative L2), or a
BF16 rounding that falls the other way (2^-8: 4e-3)."""
import numpy as np
import pytest

from dynamicradiancevolume_gb300 import abi, pipeline
from test_gpu_light_paths import _lit
from test_gpu_parity import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("width,lights,rsm,lod,sh,cap", [(1, 1, 4, 0, 1, 0), (3, 3, 128, 0, 2, 0), (40, 2, 64, 1, 2, 0),
                                                         (64, 1, 64, 0, 1, 0), (64, 1, 64, 0, 2, 100000)])
def test_gather_units_match_single_launch(width, lights, rsm, lod, sh, cap, bf16, lib, cuda):
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=width, height=width, n_lights=lights, rsm_resolution=rsm,
                        shadow_lod=lod, sh_order=sh, precision=abi.PRECISION_BF16 if bf16 else abi.PRECISION_FP32)
    p1, pos1, sh1 = _lit(w, 21, light_path=abi.LIGHT_PATH_SINGLE)
    p2, pos2, sh2 = _lit(w, 21, light_path=abi.LIGHT_PATH_SPLIT, pair_capacity=cap)
    assert np.array_equal(pos1, pos2) and len(pos1) > 0
    tol = 4e-3 if bf16 else 1e-5
    assert rel_l2(sh2, sh1) < tol
    if not bf16:
        p2.light()
        p2.sync()
        again = p2.read_entries_decoded(len(pos2))[1]
        order = np.lexsort(p2.read_entries_decoded(len(pos2))[0].T[::-1])
        assert rel_l2(again[order], 2 * sh1) < tol
    p1.close()
    p2.close()
