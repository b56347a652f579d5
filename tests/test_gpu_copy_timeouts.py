"""Stages whose copies into shared memory are withheld (DrvTuning.gather_wait_test),
so that a bounded wait runs out: the stage reports it, adds nothing that belongs
to another stage, and leaves nothing behind that a later stage reads."""
import ctypes as C

import numpy as np
import pytest

import dynamicradiancevolume_gb300 as drv
from dynamicradiancevolume_gb300 import abi, pipeline
from test_gpu_light_paths import W_MULTI_UNIT, _lit

pytestmark = pytest.mark.gpu


def _timed_out(p):
    with pytest.raises(drv.DrvError) as e:
        p.sync()
    assert e.value.status == abi.ERR_TIMEOUT


def _sorted(p, n=None):
    # n: the caches' number, where a latched error keeps drv_get_cache_count from giving it
    pos, sh = p.read_entries_decoded(p.cache_count() if n is None else n)
    order = np.lexsort(pos.T[::-1])
    return pos[order], sh[order]


@pytest.mark.parametrize("spec", [0, 8])
@pytest.mark.parametrize("bf16", [False, True])
def test_cull_copy_timeout_lists_nothing(bf16, spec, lib, cuda):
    """A cull whose records never arrive lists no pairs, so the stage adds no
    light: the runs of the context's stage before (another scene, three lights)
    are not taken for this one's. Lit again, the caches are those of a context
    that never timed out, bit for bit."""
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=96, height=64, n_lights=3, rsm_resolution=32,
                        specular_envmap_size=spec, precision=abi.PRECISION_BF16 if bf16 else abi.PRECISION_FP32)
    p = pipeline.Pipeline(pipeline.host_frame(w, 3))
    p.set_tuning(light_path=abi.LIGHT_PATH_SPLIT)

    def prepare(seed, wait_test):
        p.set_frame(pipeline.host_frame(w, seed))
        p.set_tuning(gather_wait_test=wait_test)
        p.raycast_inputs()
        p.prepare_and_extract()
        p.voxelize()
        p.allocate()

    def light_one():
        assert lib.drv_light_caches(p.ctx, p.hf.lights, 1, C.byref(p.hf.volume), C.byref(p.hf.frame)) == abi.OK

    prepare(4, 0)
    light_one()
    p.sync()
    ref = _sorted(p)
    assert ref[1].any()
    prepare(3, 0)
    p.light()
    p.sync()
    prepare(4, 2)
    light_one()
    _timed_out(p)
    assert p.light_pairs() == 0
    pos, sh = _sorted(p, len(ref[0]))
    assert np.array_equal(pos, ref[0]) and not sh.any()
    if spec:
        assert not p.read_specular(len(pos))[:, :spec * spec].any()
    prepare(4, 0)
    light_one()
    p.sync()
    got = _sorted(p)
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
    p.close()


@pytest.mark.parametrize("bf16", [False, True])
def test_stage_after_a_gather_timeout_adds_every_unit(bf16, lib, cuda):
    """The error word keeps a timeout until the next allocation. A stage that
    runs well after one that timed out (no allocation between them) adds every
    cache's light, also that of caches of several units: the timed-out stage
    added nothing, so the SH are those of one clean stage, bit for bit."""
    w = pipeline.scaled(W_MULTI_UNIT, precision=abi.PRECISION_BF16 if bf16 else abi.PRECISION_FP32)
    ref_p, ref_pos, ref_sh = _lit(w, 2, light_path=abi.LIGHT_PATH_SPLIT)
    assert ref_p.light_pairs() > 512 * ref_p.cache_count()  # caches of several units
    p = pipeline.Pipeline(pipeline.host_frame(w, 2))
    p.set_tuning(light_path=abi.LIGHT_PATH_SPLIT, gather_wait_test=1)
    p.raycast_inputs()
    p.prepare_and_extract()
    p.voxelize()
    p.allocate()
    p.light()
    _timed_out(p)
    assert not _sorted(p, len(ref_pos))[1].any()
    p.set_tuning(gather_wait_test=0)
    p.light()
    _timed_out(p)  # still latched
    pos, sh = _sorted(p, len(ref_pos))
    assert np.array_equal(pos, ref_pos) and np.array_equal(sh, ref_sh)
    p.close()
    ref_p.close()
