"""FP32 precision: the mip levels whose texels FP16 does not hold exactly are
sampled from FP32 records of the same texels, so the light stage gives the
same SH bit for bit as reading the plain mips, from the smallest grid (two
such levels) up, with a wide aperture so that the cones reach the top levels."""
import numpy as np
import pytest

from dynamicradiancevolume_gb300 import pipeline
from test_gpu_light_paths import _lit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("voxels,shadow_lod", [(32, 2), (64, 3), (256, 3), (512, 2)])
def test_wide_records_equal_plain_mips(voxels, shadow_lod, cuda, lib):
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=96, height=80, voxel_res=voxels, shadow_lod=shadow_lod,
                        max_cone_steps=32, sh_order=2, max_caches=8192)
    p1, pos1, sh1 = _lit(w, 3)
    p2, pos2, sh2 = _lit(w, 3, plain_voxel_reads=1)
    assert np.array_equal(pos1, pos2)
    assert np.abs(sh1).max() > 0
    assert np.array_equal(sh1, sh2)
    p1.close()
    p2.close()
