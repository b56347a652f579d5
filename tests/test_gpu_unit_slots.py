"""The gather's unit slots: room for units of 512 pairs and one more per cache, not
for units of 64, and a frame whose rule would list more units than that (blocks of
16 VPLs, a list about half full) takes longer ones. FP32 sums of a few hundred
thousand products in another order than the single launch's: a lane adds some
thousands of them one after the other (2e-5 relative L2)."""
import ctypes as C

import numpy as np
import pytest

from dynamicradiancevolume_gb300 import abi, pipeline
from test_gpu_light_paths import _lit
from test_gpu_parity import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [abi.PRECISION_FP32, abi.PRECISION_BF16], ids=["f32", "bf16"])
def test_context_memory_per_cache(prec, lib, cuda):
    """Device memory a context takes per additional cache: 256 pairs of 17 bytes, 1.5
    unit slots of 124 bytes, its run and unit range, its entry, an atlas of equal
    size: 4.6 KB, to the allocator's 2 MB pages."""
    import torch

    def used(max_caches):
        w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=8, height=8, max_caches=max_caches, precision=prec)
        cfg = pipeline.host_frame(w, 1).config
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        ctx = C.c_void_p()
        assert lib.drv_create(C.byref(cfg), C.byref(ctx)) == abi.OK
        got = before - torch.cuda.mem_get_info()[0]
        lib.drv_destroy(ctx)
        return got

    used(65536)  # the library's own first allocations
    per_cache = (used(262144) - used(131072)) / 131072.0
    entry = 128 if prec == abi.PRECISION_FP32 else 64
    assert per_cache <= 256 * 17 + 1.5 * 124 + 16 + entry + 32


def test_units_fit_their_slots(lib, cuda):
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], n_boxes=0, width=2, height=2, rsm_resolution=1024,
                        shadow_lod=2, max_cone_steps=1, max_caches=64)
    p1, pos1, sh1 = _lit(w, 3, light_path=abi.LIGHT_PATH_SPLIT)
    pairs, slots = p1.light_pairs(), (1 << 22) // 512 + 1 + 64  # the smallest list: 2^22 pairs
    assert pairs <= 1 << 22 and pairs / 64 > slots, (pairs, slots)
    p2, pos2, sh2 = _lit(w, 3, light_path=abi.LIGHT_PATH_SINGLE)
    assert np.array_equal(pos1, pos2) and len(pos1) > 0
    assert rel_l2(sh1, sh2) < 2e-5
    p1.close()
    p2.close()
