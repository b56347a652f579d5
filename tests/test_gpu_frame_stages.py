"""drv_frame against the stages called one by one, where the frame's launches
overlap: the light stage's tail, the specular gather, the envmaps' preparation
and the apply (its tensor-core form too), which in the stages' calls follow each
other. Frames of three scenes run back to back on one context, without a
synchronisation between them, so that a kernel that reads too early finds the
previous frame's values. Both sides add the same terms in the same order (the
gather's units follow from the frame's pairs): BF16 results and the envmaps'
R11G11B10 texels are the same bit for bit, FP32 radiance to 1e-5 relative L2."""
import numpy as np
import pytest

from dynamicradiancevolume_gb300 import abi, pipeline
from test_gpu_parity import rel_l2

pytestmark = pytest.mark.gpu

SEEDS = (11, 12, 13)


def _rough_metal(p, seed):
    rm = np.random.default_rng(seed).integers(0, 256, tuple(p.rough_metal.shape), np.uint8)
    p.rough_metal.copy_(p.torch.from_numpy(rm))


def _envmaps(p):
    n = p.cache_count()
    pos, _ = p.read_entries_decoded(n)
    return p.read_specular(n)[np.lexsort(pos.T[::-1])]


CASES = [dict(spec=8), dict(spec=16, lights=3), dict(spec=16, lights=3, fill=2), dict(spec=8, lights=3, shadow=0),
         dict(spec=8, lights=3, per_light=1), dict(spec=16, bf16=1), dict(spec=8, single=1), dict(bf16=1),
         dict(bf16=1, lights=3, per_light=1), dict(bf16=1, shadow=0), dict(bf16=1, tensor_core=1),
         dict(bf16=1, tensor_core=1, sh=2, lights=3), dict(bf16=1, tensor_core=1, shadow=0)]


@pytest.mark.parametrize("size", [(101, 67), (640, 360)], ids=["small", "large"])
@pytest.mark.parametrize("case", CASES, ids=["-".join("%s%d" % kv for kv in c.items()) for c in CASES])
def test_frames_match_their_stages(case, size, lib, cuda):
    c = dict(dict(spec=0, lights=1, shadow=1, per_light=0, bf16=0, tensor_core=0, sh=1, single=0, fill=0), **case)
    w = pipeline.scaled(pipeline.WORKLOADS["c1_small"], width=size[0], height=size[1], n_lights=c["lights"],
                        rsm_resolution=16, indirect_shadow=c["shadow"], specular_envmap_size=c["spec"],
                        specular_fill_level=c["fill"], sh_order=c["sh"],
                        precision=abi.PRECISION_BF16 if c["bf16"] else abi.PRECISION_FP32)
    knobs = dict(per_light_dispatch=c["per_light"], tensor_core_apply=c["tensor_core"],
                 light_path=abi.LIGHT_PATH_SINGLE if c["single"] else abi.LIGHT_PATH_AUTO)
    frames = [pipeline.host_frame(w, s) for s in SEEDS]
    p = pipeline.Pipeline(frames[0])
    p.set_tuning(**knobs)
    _rough_metal(p, 1)
    p.torch.cuda.synchronize()
    refs = []
    for hf in frames:
        p.set_frame(hf)
        p.raycast_inputs()
        p.prepare_and_extract()
        p.voxelize()
        p.allocate()
        p.light()
        if c["spec"]:
            p.prepare_specular()
        p.apply()
        p.sync()
        refs.append((p.out.cpu().numpy().copy(), _envmaps(p) if c["spec"] else None))
    q = pipeline.Pipeline(frames[0])
    q.set_tuning(**knobs)
    _rough_metal(q, 1)
    outs = [q.torch.full_like(q.out, 7.0) for _ in frames]
    q.torch.cuda.synchronize()
    for last in range(len(frames)):
        order = [(last + 1 + k) % len(frames) for k in range(len(frames))]  # ends with frame `last`
        for k in order:
            q.set_frame(frames[k])
            q.raycast_inputs()
            q.frame(outs[k])
        q.sync()
        for k in order:
            got, ref = outs[k].cpu().numpy(), refs[k][0]
            assert np.abs(ref).max() > 0
            if c["bf16"]:
                assert np.array_equal(got, ref)
            else:
                assert rel_l2(got, ref) < 1e-5
        if c["spec"]:
            got = _envmaps(q)
            assert got.any() and np.array_equal(got, refs[last][1])
    p.close()
    q.close()
